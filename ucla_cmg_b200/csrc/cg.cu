// cg.cu -- one Crank-Nicolson half diffusion step as a single persistent
// cooperative launch.
//
// Reference: EP_CrankNicholson::Solve (Solvers/EP_CrankNicholson.cc:99-104,
// 146-150): b = B V (B = C_m M - dt/4 K), then AztecOO CG with a Jacobi
// preconditioner on A = C_m M + dt/4 K from x0 = V, stopped when
// ||r_k||_2 <= tol ||r_0||_2.
//
// Layout: SELL-32 (slices of 32 consecutive rows, column-major inside the
// slice, one warp per slice, one lane per row) so every value/column load is
// a coalesced 128-byte transaction.  A and B share the column array.
//
// One grid barrier per iteration (k_cn_two, for matrices that stream from DRAM,
// has two).  Neighbours see a node's (z, w), z = dinv r
// and w = dinv A p, double-buffered; p, q = A p and the correction d = x - V are
// the owner's alone.  One sweep of an iteration rebuilds, for every column it
// gathers, the neighbour's new z' = z - alpha w (an explicit fma, so the owner
// and every neighbour round alike), forms u = A z' and on the own row
//   p' = z' + beta p,  q' = u + beta q  (= A p'),  w' = dinv q',  d + alpha p
// and writes (z', w') to the other buffer; nothing of the old buffer changes
// during the sweep.  (Gathering p as well and forming A p' directly took twice
// the bytes a neighbour: at 16 bytes a record a sweep is bound by L1, 2600
// cycles for 16 slices.)  alpha and beta come from one reduction at the end of
// the sweep: besides (p', q') and the residual's own (r, z), (r, r) it sums the
// products that give the next residual's,
//   (r, z)_next = (r, z) - 2 alpha d(z, w) + alpha^2 d(w, w)   (d = diag A)
// and (r, r)_next likewise.  Both start from sums of the vectors themselves
// in every sweep, so the differences (one iteration's reduction, a factor of
// ten or so, out of FP64's sixteen digits) do not accumulate: the iterates
// and the stop test are those of the two-reduction recurrences to rounding.
// The second sweep and second barrier of those (x, r, z updated after alpha
// is known) cost 12 us a phase with 888 CTAs polling one counter, which was
// most of a solve's time on every mesh under a million nodes.
// Gathers are plain (L1-allocating) loads: the barrier's acquire orders every
// block's writes of the previous sweep before them, and the rows of a slice
// share many neighbours.
// Dot products accumulate in FP64 whatever the vector type.  Reductions
// sum the per-block partials in block order, so results are deterministic.
#include <algorithm>

#include "kernels.cuh"

namespace ep {

__device__ __forceinline__ float ldcg(const float *p) { return __ldcg(p); }
__device__ __forceinline__ double ldcg(const double *p) { return __ldcg(p); }

// What neighbours read of a node, (z, w), in one load.
template <typename R> struct Pair { R z, w; };
__device__ __forceinline__ Pair<float> pair_load(const float *q, int i) {
    const float2 t = reinterpret_cast<const float2 *>(q)[i];
    return {t.x, t.y};
}
__device__ __forceinline__ Pair<double> pair_load(const double *q, int i) {
    const double2 t = reinterpret_cast<const double2 *>(q)[i];
    return {t.x, t.y};
}
__device__ __forceinline__ void pair_store(float *q, int i, float z, float w) {
    reinterpret_cast<float2 *>(q)[i] = make_float2(z, w);
}
__device__ __forceinline__ void pair_store(double *q, int i, double z, double w) {
    reinterpret_cast<double2 *>(q)[i] = make_double2(z, w);
}
// a gathered node's new z
template <typename R>
__device__ __forceinline__ R pair_z(const R *q, int c, R alpha) {
    const Pair<R> t = pair_load(q, c);
    return fma(-alpha, t.w, t.z);
}
// what only the owner reads of a row: p, q = A p, d = x - V
template <typename R> struct Own { R p, q, d; };
template <typename R>
__device__ __forceinline__ Own<R> own_load(const CGArgs<R> &a, int i) { return {a.po[i], a.qo[i], a.dc[i]}; }
template <typename R>
__device__ __forceinline__ void own_store(const CGArgs<R> &a, int i, R p, R q, R d) {
    a.po[i] = p; a.qo[i] = q; a.dc[i] = d;
}

// A row's terms of the seven sums (see the top).
template <typename R>
__device__ __forceinline__ void row_sums(double d, R z, R w, R p, R q, double (&v)[7]) {
    const double dz = d * (double)z, dw = d * (double)w;
    v[0] += (double)p * (double)q;
    v[1] += dz * (double)z;
    v[2] += dz * (double)w;
    v[3] += dw * (double)w;
    v[4] += dz * dz;
    v[5] += dz * dw;
    v[6] += dw * dw;
}

// One row of a sweep, with u = A z' of it: the new vectors and the sums.
template <typename R>
__device__ __forceinline__ void sweep_row(const CGArgs<R> &a, R *nxt, int row, R di, const Pair<R> &t, const Own<R> &o,
                                          R u, R al, R be, double (&v)[7]) {
    const R z = fma(-al, t.w, t.z), p = fma(be, o.p, z), q = fma(be, o.q, u), w = di * q;
    pair_store(nxt, row, z, w);
    own_store(a, row, p, q, fma(al, o.p, o.d));
    row_sums((double)(R(1) / di), z, w, p, q, v);
}

// ---- grid barrier and reduction in one ----
// Every CTA of a group publishes its partial sums as 16-byte {value, tag}
// units (one 128-byte line per CTA) and then reads every other CTA's line
// until the tags are this phase's: one store and one load round trip, where
// a counter barrier followed by a read of the partials takes an atomic, a
// generation poll and a read.  A unit is one 128-bit access, so a value
// never comes with another phase's tag.  Two sets of lines alternate: a CTA
// writes set s again only after the next phase's tags of everybody, which
// nobody publishes before it has read set s.  Tags go on from launch to
// launch (GridBarrier::seq), so a line never holds a tag of the future.
// Waits are bounded as in grid_sync.  A group of one CTA needs no global
// memory at all.
constexpr int kRedMax = 8;                    // values of one reduction, at most
__device__ __forceinline__ void slot_store(CgSlot *p, double v, unsigned long long tag) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"((unsigned long long)__double_as_longlong(v)), "l"(tag)
                 : "memory");
}
__device__ __forceinline__ void slot_load(const CgSlot *p, double &v, unsigned long long &tag) {
    unsigned long long u;
    asm volatile("{\n\t.reg .b128 t;\n\tld.acquire.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(u), "=l"(tag)
                 : "l"(p)
                 : "memory");
    v = __longlong_as_double((long long)u);
}
__device__ __forceinline__ void fence_acq_rel_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// A warp's sums of NV <= 8 values: each step halves the values a lane carries, so
// lane l ends with value l / 4 (18 shuffles for 8 FP64 sums instead of 80).
template <int NV>
__device__ __forceinline__ double warp_sums(const double (&vin)[NV]) {
    const int lane = threadIdx.x & 31;
    double v[kRedMax];
#pragma unroll
    for (int k = 0; k < kRedMax; k++) v[k] = k < NV ? vin[k < NV ? k : 0] : 0.0;
#pragma unroll
    for (int st = 0; st < 3; st++) {
        const int half = 4 >> st, o = 16 >> st;
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < half; i++) {
            const double send = up ? v[i] : v[i + half], keep = up ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
    return v[0];
}
// value lane & 7 summed over the rows of a [rows][8] array, on every lane
__device__ __forceinline__ double column_sum(const double (*sh)[kRedMax], int rows) {
    const int lane = threadIdx.x & 31;
    double t = 0.0;
    for (int r = lane >> 3; r < rows; r += 4) t += sh[r][lane & 7];
    t += __shfl_xor_sync(0xffffffffu, t, 8);
    t += __shfl_xor_sync(0xffffffffu, t, 16);
    return t;
}

// A group of many CTAs (a launch shape set by the caller): every CTA reading
// every line is nb^2 reads (1184 CTAs of 128 threads, 28.6K nodes FP32: 670 us
// of CG a step), so every 32nd CTA adds its 32 lines first and the others read
// those sums, one more round trip (205 us; 592 of 256 threads 255 -> 183).
// `lines` lines from `line` on, their sum to `sum`.  Not inlined: its registers
// are not the sweep's (and the gather width 4 has an instance without it, WIDE
// false, which 781K nodes run 10 % faster at 148 CTAs).
constexpr int kRedFlat = 296, kRedGroup = 32;
__device__ __noinline__ bool add_lines(const CgSlot *line, CgSlot *sum, int lines, int nv, unsigned long long tag,
                                       GridBarrier *bar, unsigned int lim) {
    __shared__ double sh[32][kRedMax];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int polls = 0;
    int bad = 0;
    double acc = 0.0;
    for (int u = threadIdx.x; u < lines * kRedMax && (u & (kRedMax - 1)) < nv && !bad; u += blockDim.x) {
        double x;
        unsigned long long t;
        for (slot_load(line + u, x, t); t != tag; slot_load(line + u, x, t)) {
            if (++polls > lim) { atomicExch(&bar->err, 1u); bad = 1; break; }
            if ((polls & 15u) == 0) {
                if (*(volatile unsigned int *)&bar->err) { bad = 1; break; }
                __nanosleep(64);
            }
        }
        acc += x;
    }
    acc += __shfl_xor_sync(0xffffffffu, acc, 8);
    acc += __shfl_xor_sync(0xffffffffu, acc, 16);
    if (lane < kRedMax) sh[warp][lane] = acc;
    if (__syncthreads_or(bad)) return false;
    if (warp == 0) {
        const double t = column_sum(sh, blockDim.x >> 5);
        fence_acq_rel_gpu();                  // what the CTAs released before their sum's tag
        if (lane < nv) slot_store(sum + lane, t, tag);
    }
    return true;
}

// NV <= 8 sums over the CTAs [b0, b0 + nb) of a group, the same bits in every
// thread of every CTA, and a barrier between what the group wrote before and
// what it reads after.  false: a wait gave up, here or (ok false) before.
template <int NV, bool WIDE = false>
__device__ __forceinline__ bool group_reduce(CgSlot *slots, int G, unsigned long long tag, int b0, int nb,
                                             unsigned int hold, GridBarrier *bar, const double (&vin)[NV],
                                             double (&tot)[NV], bool ok = true) {
    static_assert(NV <= kRedMax, "too many values");
    __shared__ double sh_a[32][kRedMax], sh_b[32][kRedMax];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const double own = warp_sums(vin);
    if ((lane & 3) == 0) sh_a[warp][lane >> 2] = own;
    __syncthreads();
    double t;
    if (nb == 1 && !hold) {
        t = column_sum(sh_a, nw);
        if (__syncthreads_or(!ok)) {          // sh_a is free again
            if (tid == 0) atomicExch(&bar->err, 1u);
            return false;
        }
    } else {
        CgSlot *set = slots + (size_t)(tag & 1) * G * kRedMax;
        if (warp == 0) {
            const double mine = column_sum(sh_a, nw);
            fence_acq_rel_gpu();              // the CTA's writes (ordered here by the CTA barrier) before the tag
            if (lane < NV) slot_store(set + (size_t)blockIdx.x * kRedMax + lane, mine, tag);
        }
        const unsigned int lim = bar->limit ? bar->limit : kGridPolls;
        const CgSlot *grp = set + (size_t)b0 * kRedMax;
        int units = nb * kRedMax, every = 1;  // the lines to read, `every` lines apart
        if (WIDE && nb > kRedFlat) {
            const int k = (int)blockIdx.x - b0;
            CgSlot *sums = set + (size_t)2 * G * kRedMax;
            if (k % kRedGroup == 0 && !add_lines(grp + (size_t)k * kRedMax, sums + (size_t)blockIdx.x * kRedMax,
                                                 min(kRedGroup, nb - k), NV, tag, bar, lim))
                return false;
            grp = sums + (size_t)b0 * kRedMax;
            units = (nb + kRedGroup - 1) / kRedGroup * kRedMax;
            every = kRedGroup;
        }
        auto unit = [&](int u) { return grp + (WIDE ? u + (u / kRedMax) * (every - 1) * kRedMax : u); };
        const bool mine = (tid & (kRedMax - 1)) < NV;
        unsigned int polls = 0;
        int bad = ok ? 0 : 1;
        if (bad) atomicExch(&bar->err, 1u);
        double acc = 0.0;
        for (int u0 = tid; u0 < units && mine && !bad; u0 += 4 * (int)blockDim.x) {
            double x[4];
            unsigned int pend = 0;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                x[i] = 0.0;
                if (u0 + i * (int)blockDim.x < units) pend |= 1u << i;
            }
            if (hold) pend |= 16u;            // arrivals that never come (ep_test_hold_barrier)
            while (pend) {
                unsigned long long tg[4];
                double xv[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (pend >> i & 1u) slot_load(unit(u0 + i * (int)blockDim.x), xv[i], tg[i]);
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if ((pend >> i & 1u) && tg[i] == tag) { x[i] = xv[i]; pend &= ~(1u << i); }
                if (pend) {
                    if (++polls > lim) { atomicExch(&bar->err, 1u); bad = 1; break; }
                    if ((polls & 15u) == 0) {
                        if (*(volatile unsigned int *)&bar->err) { bad = 1; break; }
                        __nanosleep(64);
                    }
                }
            }
            acc += (x[0] + x[1]) + (x[2] + x[3]);
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 8);
        acc += __shfl_xor_sync(0xffffffffu, acc, 16);
        if (lane < kRedMax) sh_b[warp][lane] = acc;
        if (__syncthreads_or(bad)) return false;
        t = column_sum(sh_b, nw);
    }
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = __shfl_sync(0xffffffffu, t, k);
    return true;
}

template <int NV>
__device__ __forceinline__ void block_reduce_store(double (&v)[NV], double *out, int stride) {
    __shared__ double sh[NV][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) sh[k][warp] = v[k];
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double t = lane < nw ? sh[k][lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) out[k * stride + blockIdx.x] = t;
        }
    }
    __syncthreads();
}

// every block of a group sums the group's partials in the same order
template <int NV>
__device__ __forceinline__ void grid_total(const double *partial, int stride, int b0, int nblk, double (&tot)[NV]) {
    __shared__ double sh[NV];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double t = 0.0;
            for (int b = lane; b < nblk; b += 32) t += __ldcg(partial + k * stride + b0 + b);
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) sh[k] = t;
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = sh[k];
    __syncthreads();
}

// Ask L2 for the column indices and values (and the B values when Bv is
// given) of slice sn, which this warp reads next: one lane issues bulk L2
// prefetches, so the warp's next index loads hit L2 instead of waiting on
// DRAM.  A hint only: nothing waits on it.  Every slice starts on a 128-byte
// boundary of the arrays and spans a multiple of 128 bytes.
__device__ __forceinline__ void l2_prefetch(const void *p, unsigned bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
template <typename R>
__device__ __forceinline__ void prefetch_slice(const int *__restrict__ slice_ptr, const int *col, const R *Av,
                                               const R *Bv, int sn, int s_hi, int lane) {
    if (lane == 0 && sn < s_hi) {
        const int b = slice_ptr[sn], e = slice_ptr[sn + 1];
        if (e > b) {
            l2_prefetch(col + b, (unsigned)(e - b) * 4u);
            l2_prefetch(Av + b, (unsigned)(e - b) * (unsigned)sizeof(R));
            if (Bv) l2_prefetch(Bv + b, (unsigned)(e - b) * (unsigned)sizeof(R));
        }
    }
}

// The columns k .. w-1 (fewer than NB) of a slice as one group: loads of the
// columns that exist (the test is the same for the whole warp), then their
// gathers, then the products added in column order.
template <int NB, typename R, typename F>
__device__ __forceinline__ R slice_tail(const int *__restrict__ col, const R *__restrict__ val, int beg, int k, int w,
                                        int lane, F gather, R acc) {
    int c[NB];
    R v[NB], g[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) {
        if (k + u < w) {
            const int idx = beg + (k + u) * kSlice + lane;
            c[u] = __ldg(col + idx);
            v[u] = __ldg(val + idx);
        }
    }
#pragma unroll
    for (int u = 0; u < NB; u++)
        if (k + u < w) g[u] = gather(c[u]);
#pragma unroll
    for (int u = 0; u < NB; u++)
        if (k + u < w) acc += v[u] * g[u];
    return acc;
}

// G columns k .. k+G-1 of a slice as one group: their column and value loads,
// then their gathers, then the products added in column order
template <int G, typename R, typename F>
__device__ __forceinline__ R slice_group(const int *__restrict__ col, const R *__restrict__ val, int beg, int k,
                                         int lane, F gather, R acc) {
    int c[G];
    R v[G], g[G];
#pragma unroll
    for (int u = 0; u < G; u++) {
        const int idx = beg + (k + u) * kSlice + lane;
        c[u] = __ldg(col + idx);
        v[u] = __ldg(val + idx);
    }
#pragma unroll
    for (int u = 0; u < G; u++) g[u] = gather(c[u]);
#pragma unroll
    for (int u = 0; u < G; u++) acc += v[u] * g[u];
    return acc;
}

// Row sums of one SELL slice, NB slice columns at a time: the column and
// value loads of a group are issued together, then the gathers, so each lane
// has 3 NB independent loads in flight (at one lane per row the kernel is
// bound by memory latency, not bandwidth); the w mod NB columns left over
// form one more, partial group -- except a single one, which joins the last
// full group (a 17-wide slice gathers in 2 rounds of 8 + 9, not 3 of
// 8 + 8 + 1: on the shell's meshes this is what evens out the warps' loads).
// The products are still added in column order, so the sums are those of
// the plain loop whatever the grouping.
template <int NB, typename R, typename F>
__device__ __forceinline__ R slice_row_sum(const int *__restrict__ col, const R *__restrict__ val, int beg, int w,
                                           int lane, F gather) {
    R acc = R(0);
    int k = 0;
    for (; k + NB <= w && w - k != NB + 1; k += NB) acc = slice_group<NB>(col, val, beg, k, lane, gather, acc);
    if (w - k == NB + 1) acc = slice_group<NB + 1>(col, val, beg, k, lane, gather, acc);
    else if (k < w) acc = slice_tail<NB>(col, val, beg, k, w, lane, gather, acc);
    return acc;
}

// Prologue sums of one slice row: A x and B x, and A d when pred (d = the
// predictor's start correction, dget(c) its value at column c), NB columns
// a group like slice_row_sum; each sum is added in column order.
template <int NB, typename R, typename FD>
__device__ __forceinline__ void slice_ab_sums(const int *__restrict__ col, const R *__restrict__ Av,
                                              const R *__restrict__ Bv, const R *x, int beg, int w, int lane,
                                              bool pred, FD dget, R &ax, R &bx, R &ad) {
    for (int k = 0; k < w; k += NB) {
        int c[NB];
        R av[NB], bv[NB], xv[NB], dv[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) {
            if (k + u < w) {
                const int idx = beg + (k + u) * kSlice + lane;
                c[u] = __ldg(col + idx);
                av[u] = __ldg(Av + idx);
                bv[u] = __ldg(Bv + idx);
            }
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            if (k + u < w) {
                xv[u] = x[c[u]];
                if (pred) dv[u] = dget(c[u]);
            }
        }
#pragma unroll
        for (int u = 0; u < NB; u++) {
            if (k + u < w) {
                ax += av[u] * xv[u];
                bx += bv[u] * xv[u];
                if (pred) ad += av[u] * dv[u];
            }
        }
    }
}

// The same sum with the next group's column and value loads issued before
// the current group's gathers (software pipelining: the index loads of
// group k + 1 overlap the gathers of group k).  Same order of additions.
template <int NB, typename R, typename F>
__device__ __forceinline__ R slice_row_sum_pipe(const int *__restrict__ col, const R *__restrict__ val, int beg, int w,
                                                int lane, F gather) {
    R acc = R(0);
    const int full = w / NB;
    int c[NB], cn[NB];
    R v[NB], vn[NB];
    if (full > 0) {
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int idx = beg + u * kSlice + lane;
            c[u] = __ldg(col + idx);
            v[u] = __ldg(val + idx);
        }
    }
    for (int b = 0; b < full; b++) {
        const bool more = b + 1 < full;
#pragma unroll
        for (int u = 0; u < NB; u++) {
            const int idx = beg + ((b + 1) * NB + u) * kSlice + lane;
            cn[u] = more ? __ldg(col + idx) : 0;
            vn[u] = more ? __ldg(val + idx) : R(0);
        }
        R g[NB];
#pragma unroll
        for (int u = 0; u < NB; u++) g[u] = gather(c[u]);
#pragma unroll
        for (int u = 0; u < NB; u++) acc += v[u] * g[u];
#pragma unroll
        for (int u = 0; u < NB; u++) { c[u] = cn[u]; v[u] = vn[u]; }
    }
    if (full * NB < w) acc = slice_tail<NB>(col, val, beg, full * NB, w, lane, gather, acc);
    return acc;
}

constexpr int kUnitCols = 8;

__host__ __device__ inline size_t unit_bytes(int rsize) { return (size_t)kUnitCols * kSlice * (4 + (size_t)rsize); }
// dynamic shared memory of a CTA of `block` threads, `depth` units in flight per warp
__host__ __device__ inline size_t stage_smem_bytes(int block, int depth, int rsize) {
    return (size_t)(block / 32) * (size_t)(depth + 1) * unit_bytes(rsize);
}

__device__ __forceinline__ uint32_t cg_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

// one 16-byte global -> shared copy, cached in L2 only (both addresses
// 16-byte aligned: every unit starts on a 128-byte boundary of the SELL
// arrays and of the ring)
__device__ __forceinline__ void cp16(void *dst, const void *src, uint64_t pol) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(cg_smem_u32(dst)), "l"(src),
                 "l"(pol)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// this thread's copies of every unit but the newest depth - 1 have landed
__device__ __forceinline__ void unit_wait(int depth) {
    switch (depth) {
        case 1: cp_wait<0>(); break;
        case 2: cp_wait<1>(); break;
        case 3: cp_wait<2>(); break;
        default: cp_wait<3>(); break;
    }
}

template <typename R>
struct UnitRing {
    int *idx;          // slot k's indices at idx + k * kUnitCols * kSlice
    R *val;            // slot k's values at val + k * kUnitCols * kSlice
    int slots, depth;  // slots = depth + 1
    int L;             // this warp's slices per sweep (0: nothing to stage)
    int j, k, beg, w;  // producer cursor: slice j of the warp, its column k, start, width
    int issued;        // units issued so far
    uint64_t pol;
};

// issue the unit under the cursor into the ring slot of its position and
// advance the cursor (the next unit of the slice, or the next slice,
// wrapping to the warp's first slice: the next sweep).  Every lane commits
// one copy group per call, empty or not, so the group counts stay uniform.
template <typename R>
__device__ __forceinline__ void unit_issue(UnitRing<R> &q, const CGArgs<R> &a, int gwarp, int nwarps, int lane) {
    if (q.L > 0) {
        const int slot = q.issued % q.slots;
        const int nc = min(kUnitCols, q.w - q.k);
        int *di = q.idx + slot * (kUnitCols * kSlice);
        R *dv = q.val + slot * (kUnitCols * kSlice);
        const int *si = a.col + q.beg + q.k * kSlice;
        const R *sv = a.Aval + q.beg + q.k * kSlice;
        // indices: column u, 16-byte piece p is chunk c = 8 u + p
#pragma unroll
        for (int t = 0; t < 2; t++) {
            const int c = lane + 32 * t;
            if ((c >> 3) < nc) cp16(di + 4 * c, si + 4 * c, q.pol);
        }
        // values: VPC chunks of VE values per column
        constexpr int VPC = kSlice * (int)sizeof(R) / 16, VE = 16 / (int)sizeof(R);
#pragma unroll
        for (int t = 0; t < VPC * kUnitCols / 32; t++) {
            const int c = lane + 32 * t;
            if (c / VPC < nc) cp16(dv + VE * c, sv + VE * c, q.pol);
        }
        q.k += kUnitCols;
        while (q.k >= q.w) {               // ends: some slice of the warp has columns (q.L > 0)
            q.j = q.j + 1 == q.L ? 0 : q.j + 1;
            const int s = gwarp + q.j * nwarps;
            q.beg = __ldg(a.slice_ptr + s);
            q.w = (__ldg(a.slice_ptr + s + 1) - q.beg) / kSlice;
            q.k = 0;
        }
    }
    q.issued++;
    cp_commit();
}

// the warp's ring and its cursor at the first unit
template <typename R>
__device__ __forceinline__ void ring_start(UnitRing<R> &q, const CGArgs<R> &a, unsigned char *sm, int gwarp, int nwarps,
                                           int s_hi) {
    q.depth = a.depth;
    q.slots = a.depth + 1;
    // slots x unit of indices, then slots x unit of values
    unsigned char *base = sm + (size_t)(threadIdx.x >> 5) * q.slots * unit_bytes((int)sizeof(R));
    q.idx = reinterpret_cast<int *>(base);
    q.val = reinterpret_cast<R *>(base + (size_t)q.slots * kUnitCols * kSlice * 4);
    q.L = gwarp < s_hi ? (s_hi - gwarp + nwarps - 1) / nwarps : 0;
    int cols = 0;
    for (int j = 0; j < q.L; j++) {
        const int s = gwarp + j * nwarps;
        cols += __ldg(a.slice_ptr + s + 1) - __ldg(a.slice_ptr + s);
    }
    if (cols == 0) q.L = 0;
    q.j = 0;
    q.k = 0;
    q.beg = q.L > 0 ? __ldg(a.slice_ptr + gwarp) : 0;
    q.w = q.L > 0 ? (__ldg(a.slice_ptr + gwarp + 1) - q.beg) / kSlice : 0;
    while (q.L > 0 && q.w == 0) {      // ends: some slice has columns
        q.j++;
        const int s = gwarp + q.j * nwarps;
        q.beg = __ldg(a.slice_ptr + s);
        q.w = (__ldg(a.slice_ptr + s + 1) - q.beg) / kSlice;
    }
    q.issued = 0;
    q.pol = l2_evict_first_policy();
}

// the row sum of a slice of w columns out of the ring
template <typename R, typename F>
__device__ __forceinline__ R ring_row_sum(UnitRing<R> &q, const CGArgs<R> &a, int gwarp, int nwarps, int lane, int w,
                                          int &cons, F gather) {
    R acc = R(0);
    for (int k = 0; k < w; k += kUnitCols, cons++) {
        unit_wait(q.depth);
        __syncwarp();                 // the unit is visible to every lane, and every
                                      // lane is done with the slot refilled next
        unit_issue(q, a, gwarp, nwarps, lane);
        const int off = (cons % q.slots) * (kUnitCols * kSlice) + lane;
        const int *ci = q.idx + off;
        const R *cv = q.val + off;
        const int nc = min(kUnitCols, w - k);
        int c[kUnitCols];
        R g[kUnitCols];
#pragma unroll
        for (int u = 0; u < kUnitCols; u++)
            if (u < nc) c[u] = ci[u * kSlice];
#pragma unroll
        for (int u = 0; u < kUnitCols; u++)
            if (u < nc) g[u] = gather(c[u]);
#pragma unroll
        for (int u = 0; u < kUnitCols; u++)
            if (u < nc) acc += cv[u * kSlice] * g[u];
    }
    return acc;
}

// A CTA's instance (its rows [rb, re), its CTA group [b0, b0 + nb) and its
// barrier) and its slices [s0, s1): a contiguous share of the instance's, so
// that neighbouring rows share gathered values in L1; its warps take them in
// turn.
struct CgShare { int inst, b0, nb, rb, re, s0, s1; };
template <typename R>
__device__ __forceinline__ CgShare cg_share(const CGArgs<R> &a) {
    CgShare h{0, 0, (int)gridDim.x, 0, a.n, 0, 0};
    if (a.ninst > 1) {
        int lo = 0, hi = a.ninst - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.inst_blk[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
        }
        h.inst = lo;
        h.b0 = a.inst_blk[lo]; h.nb = a.inst_blk[lo + 1] - h.b0;
        h.rb = a.inst_row[lo]; h.re = a.inst_row[lo + 1];
    }
    const int lo = h.rb / kSlice, all = (h.re + kSlice - 1) / kSlice - lo, ci = (int)blockIdx.x - h.b0;
    h.s0 = lo + (int)((long long)all * ci / h.nb);
    h.s1 = lo + (int)((long long)all * (ci + 1) / h.nb);
    return h;
}

// The end of a solve: V + its correction, which is also the next solve's
// predictor (own rows), and the statistics.
template <typename R>
__device__ __forceinline__ void finish_correction(const CGArgs<R> &a, int row, R dn) {
    a.x[row] += dn;
    if (a.delta) {
        if (a.dext) a.dext[row] = R(2) * dn - a.delta[row];     // the next solve's start: 2 delta - delta_prev
        a.delta[row] = dn;
    }
}
// (the last step's alpha p is still to be added)
template <typename R>
__device__ __forceinline__ void finish_row(const CGArgs<R> &a, int row, const Pair<R> &t, const Own<R> &o, R al, R be,
                                           bool converged) {
    R dn = fma(al, o.p, o.d);
    // FP32, which stops at the resolution of b: one more step for
    // free, the next iteration's direction taken with this iteration's
    // length (successive lengths differ by a few percent on these
    // mass-dominated systems, so it lowers the error 2-3 fold, as the
    // iteration itself would).  FP64 keeps the reference's iterate.
    if (sizeof(R) == 4 && converged) dn = fma(al, fma(be, o.p, fma(-al, t.w, t.z)), dn);
    finish_correction(a, row, dn);
}
template <typename R>
__device__ __forceinline__ void finish_statistics(const CGArgs<R> &a, const CgShare &sh, bool converged,
                                                  unsigned long long tag, int it, double rr, double rr0) {
    if ((int)blockIdx.x == sh.b0 && threadIdx.x == 0) {
        a.bar[sh.inst].seq = tag;             // every CTA of the group has read the old one
        atomicAdd(a.iters_total, (unsigned long long)it);
        atomicMax(a.iters_max, (unsigned int)it);
        if (!converged) atomicAdd(a.fails, 1u);
        if (a.last) {
            a.last[2 * sh.inst] = (double)it;
            a.last[2 * sh.inst + 1] = rr0 > 0.0 ? sqrt(fmax(rr, 0.0) / rr0) : 0.0;
        }
    }
}
template <typename R>
__device__ __forceinline__ void cg_finish(const CGArgs<R> &a, const CgShare &sh, int warp, int nw, int lane,
                                          const R *cur, R al, R be, bool converged, unsigned long long tag, int it,
                                          double rr, double rr0) {
    for (int s = sh.s0 + warp; s < sh.s1; s += nw) {
        const int row = s * kSlice + lane;
        if (row >= sh.rb && row < sh.re) finish_row(a, row, pair_load(cur, row), own_load(a, row), al, be, converged);
    }
    finish_statistics(a, sh, converged, tag, it, rr, rr0);
}

// The solve.  NB: slice columns gathered together (4, 8; 16: 8 with the next
// group's indices and values loaded ahead; kStagedBatch: 8 out of a shared-
// memory ring, below).  NB = 4 has 64 registers, so one CTA of up to 1024
// threads per SM; the others, whose gathered values spill in 64, three of 256
// threads in FP32 (80 registers) and two in FP64 (128).  CG us a step of width
// 8 / 16 / staged, with four CTAs (64 registers; FP64 staged three) and now:
// FP32 214K nodes 248 / 307 / 314 -> 206 / 239 / 266, 781K 766 / 820 / 796 ->
// 760 / 792 / 694; FP64 214K 590 / 833 / 607 -> 361 / 385 / 389.
//
// The staged form takes the matrix stream of the sweeps off the warps'
// critical path.  A warp's slices are cut into units of kUnitCols slice
// columns: the column indices and A values of one slice's columns k .. k+7 (8
// x 128 bytes of indices, 8 x 32 x sizeof(R) bytes of values).  The warp
// copies the units into a ring of shared memory with per-thread asynchronous
// copies (cp.async.cg: 16 bytes each, L2 only, evict-first, so the matrix
// streams through L2 while the gathered records stay there), `depth` units
// ahead of the one it gathers for; the loads in flight occupy ring slots
// instead of registers.  The stream runs on past the end of a sweep into the
// next iteration's first units (the matrix does not change), under the
// reduction.  No wait on it spins: cp.async.wait_group is the hardware's wait
// for the thread's own copies, and every exit path waits for all of them.
// Same order of additions in every form, so the same bits on the same grid.
template <typename R, int NB, bool WIDE = NB != 4>
__global__ void __launch_bounds__(NB == 4 ? 1024 : 256, NB == 4 ? 1 : sizeof(R) == 8 ? 2 : 3)
k_cn_half(const CGArgs<R> a) {
    constexpr bool STAGED = NB == kStagedBatch;
    extern __shared__ __align__(128) unsigned char cg_sm[];
    const int lane = threadIdx.x & 31;
    const int G = gridDim.x;
    const CgShare sh = cg_share(a);
    const int inst = sh.inst, b0 = sh.b0, nb = sh.nb, rb = sh.rb, re = sh.re;
    GridBarrier *bar = a.bar + inst;
    unsigned long long tag = *(volatile unsigned long long *)&bar->seq;
    const int gwarp = sh.s0 + (int)(threadIdx.x >> 5), s_hi = sh.s1;
    const int nwarps = (int)blockDim.x >> 5;

    UnitRing<R> ring;                         // this warp's ring (staged form)
    if constexpr (STAGED) {
        ring_start(ring, a, cg_sm, gwarp, nwarps, s_hi);
        for (int d = 0; d < ring.depth; d++) unit_issue(ring, a, gwarp, nwarps, lane);
    }

    // ---- prologue: r = B x - A x, z = dinv r, p = w = 0 ----
    // With a predictor (delta: the previous solve's correction x - V of
    // this half step; with dext its linear extrapolation 2 delta - delta_prev,
    // stored by the previous solve) the iteration starts from x + pred
    // instead, r = B x - A (x + pred), while the stop test keeps the
    // reference's r0 = B x - A x.  a.x itself is written only at the end
    // (neighbours read it here).
    const bool pred = a.delta != nullptr;
    const bool lin = a.dext != nullptr;
    R *cur = a.q0, *nxt = a.q1;
    double rr0, stop2, rr_last;
    bool converged;
    {
        double v[3] = {0.0, 0.0, 0.0};
        for (int s = gwarp; s < s_hi; s += nwarps) {
            if (!STAGED && a.prefetch)
                prefetch_slice(a.slice_ptr, a.col, a.Aval, a.Bval, s + a.prefetch * nwarps, s_hi, lane);
            const int row = s * kSlice + lane;
            const int beg = a.slice_ptr[s], w = (a.slice_ptr[s + 1] - beg) / kSlice;
            R ax = R(0), bx = R(0), ad = R(0);
            slice_ab_sums<NB == 4 ? 2 : 4>(a.col, a.Aval, a.Bval, a.x, beg, w, lane, pred, [&](int c) {
                return lin ? a.dext[c] : a.delta[c];
            }, ax, bx, ad);
            if (row >= rb && row < re) {
                const R rref = bx - ax;
                const R r = pred ? rref - ad : rref;
                pair_store(cur, row, __ldg(a.dinv + row) * r, R(0));
                own_store(a, row, R(0), R(0), pred ? (lin ? a.dext[row] : a.delta[row]) : R(0));
                v[0] += (double)r * (double)r;
                v[1] += (double)bx * (double)bx;
                v[2] += (double)rref * (double)rref;
            }
        }
        double t[3];
        if (!group_reduce<3, WIDE>(a.slots, G, ++tag, b0, nb, a.bar_extra, bar, v, t)) {
            if constexpr (STAGED) cp_wait_all();
            return;
        }
        // ||r|| <= tol ||r0||, or the residual is at the resolution of b in the
        // vector type (FP32 cannot resolve a 1e-7 reduction of an r0 that is
        // itself rounding noise of B x - A x; in FP64 the floor is ~1e-16 ||b||)
        rr0 = t[2];
        stop2 = fmax(a.tol * a.tol * rr0, a.floor_rel * a.floor_rel * t[1]);
        rr_last = t[0];
        converged = t[0] <= stop2;
    }
    int it = 0, cons = 0;                     // cons: ring units consumed so far
    R al = R(0), be = R(0);
    while (!converged && it < a.maxit) {
        double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        for (int s = gwarp; s < s_hi; s += nwarps) {
            if (!STAGED && a.prefetch)
                prefetch_slice<R>(a.slice_ptr, a.col, a.Aval, nullptr, s + a.prefetch * nwarps, s_hi, lane);
            const int row = s * kSlice + lane;
            const int beg = __ldg(a.slice_ptr + s), w = (__ldg(a.slice_ptr + s + 1) - beg) / kSlice;
            auto gat = [&](int c) { return pair_z(cur, c, al); };
            R u;
            if constexpr (STAGED) u = ring_row_sum(ring, a, gwarp, nwarps, lane, w, cons, gat);
            else if constexpr (NB == 16) u = slice_row_sum_pipe<8>(a.col, a.Aval, beg, w, lane, gat);
            else u = slice_row_sum<NB>(a.col, a.Aval, beg, w, lane, gat);
            if (row >= rb && row < re)
                sweep_row(a, nxt, row, __ldg(a.dinv + row), pair_load(cur, row), own_load(a, row), u, al, be, v);
        }
        double t[7];
        if (!group_reduce<7, WIDE>(a.slots, G, ++tag, b0, nb, a.bar_extra, bar, v, t)) {
            if constexpr (STAGED) cp_wait_all();
            return;
        }
        { R *sw = cur; cur = nxt; nxt = sw; }
        // the residual this sweep started from is small enough already (the
        // test at the end of the last one could not tell): its step is not taken
        if (t[4] <= stop2) { rr_last = t[4]; converged = true; al = R(0); break; }
        const double alpha = t[1] / t[0], irz = 1.0 / t[1];       // the two divisions side by side
        const double rz = t[1] - 2.0 * alpha * t[2] + alpha * alpha * t[3];
        const double rr = t[4] - 2.0 * alpha * t[5] + alpha * alpha * t[6];
        it++;
        al = (R)alpha;
        be = (R)(rz * irz);
        rr_last = rr;
        // a non-finite residual (a NaN or inf voltage upstream) cannot
        // recover: stop now, counted as a failed solve (every block sees the
        // same total and leaves at the same iteration)
        if (!isfinite(rr)) break;
        // rr is a difference: below 1e-12 of what it came from only the next
        // sweep's own sum can tell
        converged = rr <= stop2 && stop2 >= 1e-12 * t[4];
    }
    if constexpr (STAGED) cp_wait_all();      // the units that ran ahead into the next sweep
    cg_finish(a, sh, (int)(threadIdx.x >> 5), nwarps, lane, cur, al, be, converged, tag, it, rr_last, rr0);
}

// ---------------------------------------------------------------------------
// k_cn_two: the solve in two passes an iteration, for a matrix that streams from
// DRAM.  There the reductions hardly count and what counts is how many loads are
// in flight, that is warps: a pass over the matrix with one sum (q = A p, (p, q))
// and a pass over the own rows with two ((r, z), (r, r)) run in 40 registers (gather
// width 4), 48 warps an SM, where the one-pass sweep's seven sums allow 32 at best.
// Neighbours gather (z, p) pairs; r, p', q and the correction are the owner's.  The
// group's warps take its slices in turns, so that all CTAs work on one stretch of
// the mesh at a time and L2 holds what they gather of it.  NB as in k_cn_half.
// When it runs: cg_fit and cg_named_two, with the times.

// The sums of a phase through a.partial and the counter barrier (consecutive
// phases use disjoint places, from `at` on): the tagged lines' polls would take
// the registers.
template <int NV, typename R>
__device__ __forceinline__ bool group_sums(const CGArgs<R> &a, int at, const CgShare &sh, double (&v)[NV]) {
    const int G = (int)gridDim.x;
    block_reduce_store<NV>(v, a.partial + at * G, G);
    if (!grid_sync(a.bar + sh.inst, sh.nb + a.bar_extra)) return false;
    grid_total<NV>(a.partial + at * G, G, sh.b0, sh.nb, v);
    return true;
}

template <typename R, int NB>
__global__ void __launch_bounds__(NB == 4 ? 768 : 256, NB == 4 ? 2 : (NB == kStagedBatch && sizeof(R) == 8) ? 3 : 4)
k_cn_two(const CGArgs<R> a) {
    constexpr bool STAGED = NB == kStagedBatch;
    extern __shared__ __align__(128) unsigned char cg_sm[];
    const int lane = threadIdx.x & 31;
    const CgShare sh = cg_share(a);
    // the group's warps take its slices in turns
    const int rb = sh.rb, re = sh.re, s_hi = (re + kSlice - 1) / kSlice, step = sh.nb * ((int)blockDim.x >> 5);
    const int gwarp = rb / kSlice + (((int)blockIdx.x - sh.b0) * (int)blockDim.x + (int)threadIdx.x) / 32;
    R *zp = a.q0, *rv = a.q1;

    UnitRing<R> ring;                         // this warp's ring (staged form)
    if constexpr (STAGED) {
        ring_start(ring, a, cg_sm, gwarp, step, s_hi);
        for (int d = 0; d < ring.depth; d++) unit_issue(ring, a, gwarp, step, lane);
    }

    // ---- prologue, as k_cn_half's ----
    const bool pred = a.delta != nullptr;
    double rz, rr0, stop2, rr_last;
    {
        const R *dv0 = a.dext ? a.dext : a.delta;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        for (int s = gwarp; s < s_hi; s += step) {
            if (!STAGED && a.prefetch)
                prefetch_slice(a.slice_ptr, a.col, a.Aval, a.Bval, s + a.prefetch * step, s_hi, lane);
            const int row = s * kSlice + lane;
            const int beg = a.slice_ptr[s], w = (a.slice_ptr[s + 1] - beg) / kSlice;
            R ax = R(0), bx = R(0), ad = R(0);
            slice_ab_sums<NB == 4 ? 2 : 4>(a.col, a.Aval, a.Bval, a.x, beg, w, lane, pred, [&](int c) {
                return a.dext ? a.dext[c] : a.delta[c];
            }, ax, bx, ad);
            if (row >= rb && row < re) {
                const R rref = bx - ax, r = pred ? rref - ad : rref, z = __ldg(a.dinv + row) * r;
                pair_store(zp, row, z, R(0));
                rv[row] = r;
                a.dc[row] = pred ? dv0[row] : R(0);
                v[0] += (double)r * (double)r;
                v[1] += (double)bx * (double)bx;
                v[2] += (double)rref * (double)rref;
                v[3] += (double)r * (double)z;
            }
        }
        if (!group_sums(a, 6, sh, v)) {
            if constexpr (STAGED) cp_wait_all();
            return;
        }
        rr_last = v[0];
        rr0 = v[2];
        stop2 = fmax(a.tol * a.tol * v[2], a.floor_rel * a.floor_rel * v[1]);
        rz = v[3];
    }
    bool converged = rr_last <= stop2;
    int it = 0, cons = 0;                     // cons: ring units consumed so far
    R al = R(0), be = R(0);
    while (!converged && it < a.maxit) {
        {   // p' = z + beta p, q = A p'
            double v[1] = {0.0};
            for (int s = gwarp; s < s_hi; s += step) {
                if (!STAGED && a.prefetch)
                    prefetch_slice<R>(a.slice_ptr, a.col, a.Aval, nullptr, s + a.prefetch * step, s_hi, lane);
                const int row = s * kSlice + lane;
                const int beg = __ldg(a.slice_ptr + s), w = (__ldg(a.slice_ptr + s + 1) - beg) / kSlice;
                auto gat = [&](int c) {
                    const Pair<R> t = pair_load(zp, c);
                    return fma(be, t.w, t.z);
                };
                R q;
                if constexpr (STAGED) q = ring_row_sum(ring, a, gwarp, step, lane, w, cons, gat);
                else if constexpr (NB == 16) q = slice_row_sum_pipe<8>(a.col, a.Aval, beg, w, lane, gat);
                else q = slice_row_sum<NB>(a.col, a.Aval, beg, w, lane, gat);
                if (row >= rb && row < re) {
                    const Pair<R> t = pair_load(zp, row);
                    const R p = fma(be, t.w, t.z);
                    a.po[row] = p;
                    a.qo[row] = q;
                    v[0] += (double)p * (double)q;
                }
            }
            if (!group_sums(a, 3, sh, v)) {
                if constexpr (STAGED) cp_wait_all();
                return;
            }
            al = (R)(rz / v[0]);
        }
        double v[2] = {0.0, 0.0};
        // two of the warp's slices at a time: both slices' loads go out before
        // either is updated
        for (int s = gwarp; s < s_hi; s += 2 * step) {
            const int row = s * kSlice + lane, row2 = row + step * kSlice;
            const bool on = row >= rb && row < re, on2 = s + step < s_hi && row2 >= rb && row2 < re;
            R pi = R(0), xi = R(0), ri = R(0), qi = R(0), di = R(0);
            R pi2 = R(0), xi2 = R(0), ri2 = R(0), qi2 = R(0), di2 = R(0);
            if (on) { pi = a.po[row]; xi = a.dc[row]; ri = rv[row]; qi = a.qo[row]; di = __ldg(a.dinv + row); }
            if (on2) { pi2 = a.po[row2]; xi2 = a.dc[row2]; ri2 = rv[row2]; qi2 = a.qo[row2]; di2 = __ldg(a.dinv + row2); }
            auto one = [&](int i, R p, R x, R r0, R q, R d) {
                a.dc[i] = x + al * p;
                const R r = r0 - al * q, z = d * r;
                rv[i] = r;
                pair_store(zp, i, z, p);
                v[0] += (double)r * (double)z;
                v[1] += (double)r * (double)r;
            };
            if (on) one(row, pi, xi, ri, qi, di);
            if (on2) one(row2, pi2, xi2, ri2, qi2, di2);
        }
        if (!group_sums(a, 0, sh, v)) {
            if constexpr (STAGED) cp_wait_all();
            return;
        }
        it++;
        be = (R)(v[0] / rz);
        rr_last = v[1];
        rz = v[0];
        if (!isfinite(rr_last)) break;        // as in k_cn_half
        converged = rr_last <= stop2;
    }
    if constexpr (STAGED) cp_wait_all();      // the units that ran ahead into the next pass
    for (int s = gwarp; s < s_hi; s += step) {
        const int row = s * kSlice + lane;
        if (row >= rb && row < re) {
            R dn = a.dc[row];
            if (sizeof(R) == 4 && converged) {
                const Pair<R> t = pair_load(zp, row);
                dn = fma(al, fma(be, t.w, t.z), dn);
            }
            finish_correction(a, row, dn);
        }
    }
    finish_statistics(a, sh, converged, a.bar[sh.inst].seq, it, rr_last, rr0);
}

// ---------------------------------------------------------------------------
// k_cn_smem: the solve of k_cn_half with the matrix in shared memory
// (cg_auto_shape says when).  An iteration of k_cn_half is a chain of exposed
// memory latencies (0.5-0.6 us each under load): the slice's bounds, then for
// every four columns their indices and values and then the gathers, then the
// own row, some eleven a slice.  Here the gathers are the only one: the slice
// bounds and the matrix wait in shared memory, the own row is loaded beside the
// gathers, and a slice's gathers go out together.
// Where a CTA's share of the matrix fits it is copied in once and stays for the
// whole solve; else each warp's region is a ring of units of 8 slice columns
// that bulk copies (cp.async.bulk, one lane issuing, an mbarrier per unit)
// refill as units are consumed, running on into the next sweep under the
// reduction.  A matrix that L2 does not hold streams through it sweep after
// sweep, each line gone before its next use; L2 is asked to keep the first 36
// MB of it and to pass the rest (765K nodes: 732 -> 630 us a step; 564K FP64:
// 1275 -> 968).
constexpr unsigned int kCopyPolls = 1u << 18; // tries of one unit's wait

__device__ __forceinline__ void cg_mbar_init(unsigned long long *b) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cg_smem_u32(b)) : "memory");
}
__device__ __forceinline__ void cg_mbar_expect(unsigned long long *b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cg_smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool cg_mbar_wait(unsigned long long *b, uint32_t parity) {
    for (unsigned int k = 0; k < kCopyPolls; k++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.b32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(cg_smem_u32(b)), "r"(parity)
                     : "memory");
        if (ok) return true;
    }
    return false;
}
// both addresses 16-byte aligned, bytes a multiple of 16: units start on
// 128-byte boundaries of the SELL arrays and of the region
__device__ __forceinline__ void cg_bulk(void *dst, const void *src, uint32_t bytes, unsigned long long *bar,
                                        uint64_t pol) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, "
                 "[%3], %4;" ::"r"(cg_smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(cg_smem_u32(bar)), "l"(pol)
                 : "memory");
}
// L2 policies of the ring's copies: keep, pass (l2_evict_first_policy) or none
__device__ __forceinline__ uint64_t l2_evict_last_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ uint64_t l2_normal_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}

// columns of the next unit of a slice with `rem` columns left
__device__ __forceinline__ int unit_cols(int rem) { return rem == kUnitMax ? kUnitMax : min(kUnit, rem); }

// A warp's share of the matrix in shared memory.
template <typename R>
struct MatRing {
    static constexpr int kColBytes = kSlice * (4 + (int)sizeof(R));   // one slice column
    unsigned char *base;          // the warp's region
    unsigned long long *bars;     // an mbarrier per unit slot
    const int *sp;                // slice bounds, sp[j * nw], sp[j * nw + 1]: the warp's j-th slice
    int nw, L;                    // warps of the CTA; the warp's slices
    int slots;                    // unit slots (resident: the units of the share)
    bool resident;
    int keep;                     // slices whose units L2 is asked to keep
    uint64_t pol_keep, pol_pass;
    int pj, pk, pslot, pcol;      // producer (lane 0): slice, column, slot and running column of the next unit
    int slot, ccol;               // consumer: slot and running column of the next unit
    uint32_t phase;               // and its mbarrier's parity

    // where a unit lies: packed by columns when resident, in its slot else
    __device__ __forceinline__ unsigned char *unit(int s, int col) const {
        return base + (size_t)(resident ? col : s * kUnitMax) * kColBytes;
    }
    // lane 0: copy the next unit of the share (a ring goes round and round)
    __device__ __forceinline__ void issue(const int *cols, const R *vals) {
        while (sp[pj * nw + 1] == sp[pj * nw]) next_slice();      // empty slices; the share has others
        const int beg = sp[pj * nw], w = (sp[pj * nw + 1] - beg) / kSlice;
        const int nc = unit_cols(w - pk), n = nc * kSlice;
        unsigned char *d = unit(pslot, pcol);
        unsigned long long *b = bars + pslot;
        const int *ci = cols + beg + pk * kSlice;
        const R *av = vals + beg + pk * kSlice;
        if ((((uintptr_t)ci | (uintptr_t)av) & 15u) == 0) {
            cg_mbar_expect(b, (uint32_t)nc * kColBytes);
            const uint64_t pol = pj < keep ? pol_keep : pol_pass;
            cg_bulk(d, ci, (uint32_t)n * 4u, b, pol);
            cg_bulk(d + n * 4, av, (uint32_t)n * (uint32_t)sizeof(R), b, pol);
        } else {
            // a caller's arrays that bulk copies cannot read (ep_cn_half_step_noalloc)
            for (int e = 0; e < n; e++) {
                reinterpret_cast<int *>(d)[e] = ci[e];
                reinterpret_cast<R *>(d + n * 4)[e] = av[e];
            }
            cg_mbar_expect(b, 0u);
        }
        pcol += nc;
        pk += nc;
        if (pk >= w) next_slice();
        if (++pslot == slots) pslot = 0;
    }
    __device__ __forceinline__ void next_slice() {
        pk = 0;
        if (++pj == L) { pj = 0; pcol = 0; }
    }
    // the next unit: wait for it where it has just been copied.  A wait that
    // gives up clears ok for good; the caller then reads no unit any more (its
    // indices are not there)
    __device__ __forceinline__ const unsigned char *take(int nc, bool first, bool &ok) {
        if (first || !resident) ok = ok && cg_mbar_wait(bars + slot, phase);
        const unsigned char *d = unit(slot, ccol);
        ccol += nc;
        if (++slot == slots) { slot = 0; phase ^= 1u; }
        return d;
    }
};

// Set up the warp's region and issue its first units.  sp: the CTA's slice
// bounds in shared memory; cols: columns a warp's region holds.
template <typename R>
__device__ __forceinline__ void mat_start(MatRing<R> &m, const CGArgs<R> &a, const int *sp, int nslices,
                                          unsigned char *region, unsigned long long *bars, int lane, int warp, int nw) {
    m.base = region + (size_t)warp * a.ring_cols * MatRing<R>::kColBytes;
    m.bars = bars + warp * kMaxUnits;
    m.sp = sp + warp;
    m.nw = nw;
    m.L = warp < nslices ? (nslices - warp + nw - 1) / nw : 0;
    int cols = 0, units = 0;
    for (int j = 0; j < m.L; j++) {
        const int w = (m.sp[j * nw + 1] - m.sp[j * nw]) / kSlice;
        cols += w;
        for (int k = 0; k < w; k += unit_cols(w - k)) units++;
    }
    m.resident = cols <= a.ring_cols && units <= kMaxUnits;
    m.slots = m.resident ? units : min(kMaxUnits, a.ring_cols / kUnitMax);
    m.pj = m.pk = m.pslot = m.pcol = 0;
    m.slot = m.ccol = 0;
    m.phase = 0;
    m.keep = (int)((float)m.L * a.keep);
    m.pol_keep = a.keep >= 1.0f ? l2_normal_policy() : l2_evict_last_policy();
    m.pol_pass = l2_evict_first_policy();
    if (lane == 0) {
        for (int k = 0; k < m.slots; k++) cg_mbar_init(m.bars + k);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int k = 0; k < m.slots; k++) m.issue(a.col, a.Aval);
    }
    __syncwarp();
}

// The row sum sum_k val_k gather(col_k) of the warp's next slice (w columns),
// GU units' gathers in flight together; per(k, v, g) sees every product's
// parts in column order.  Refills what it consumed.
template <typename R, int GU, typename F, typename P>
__device__ __forceinline__ void mat_slice(MatRing<R> &m, const CGArgs<R> &a, int w, bool first, int lane, bool &ok,
                                          F gather, P per) {
    using G = decltype(gather(0, 0));
    int used = 0;
    for (int k = 0; k < w;) {
        G g[GU][kUnitMax];
        const R *vp[GU];
        int nc[GU];
        int kk = k;
#pragma unroll
        for (int u = 0; u < GU; u++) {
            nc[u] = kk < w ? unit_cols(w - kk) : 0;
            if (nc[u] == 0) continue;
            const unsigned char *d = m.take(nc[u], first, ok);
            kk += nc[u];
            used++;
            if (!ok) { nc[u] = 0; continue; }
            const int *ci = reinterpret_cast<const int *>(d) + lane;
            vp[u] = reinterpret_cast<const R *>(d + nc[u] * kSlice * 4) + lane;
#pragma unroll
            for (int j = 0; j < kUnitMax; j++)
                if (j < nc[u]) g[u][j] = gather(ci[j * kSlice], kk - nc[u] + j);
        }
#pragma unroll
        for (int u = 0; u < GU; u++) {
#pragma unroll
            for (int j = 0; j < kUnitMax; j++)
                if (j < nc[u]) per(vp[u][j * kSlice], g[u][j]);
        }
        k = kk;
        if (!m.resident) {
            __syncwarp();                     // every lane is done with the units refilled now
            if (lane == 0 && ok)
                for (int u = 0; u < used; u++) m.issue(a.col, a.Aval);
            used = 0;
        }
    }
}

template <typename R, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) k_cn_smem(const CGArgs<R> a) {
    constexpr int GU = 2;                     // a slice's two units
    extern __shared__ __align__(128) unsigned char cg_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int G = gridDim.x;
    const CgShare sh = cg_share(a);
    const int b0 = sh.b0, nb = sh.nb, rb = sh.rb, re = sh.re, ns = sh.s1 - sh.s0;
    GridBarrier *bar = a.bar + sh.inst;
    unsigned long long tag = *(volatile unsigned long long *)&bar->seq;
    // dynamic shared memory: the warps' regions, their mbarriers, the slice bounds
    unsigned long long *bars =
        reinterpret_cast<unsigned long long *>(cg_sm + (size_t)nw * a.ring_cols * MatRing<R>::kColBytes);
    int *sp = reinterpret_cast<int *>(bars + nw * kMaxUnits);
    for (int k = threadIdx.x; k <= ns; k += blockDim.x) sp[k] = __ldg(a.slice_ptr + sh.s0 + k);
    __syncthreads();
    MatRing<R> m;
    mat_start(m, a, sp, ns, cg_sm, bars, lane, warp, nw);
    bool ok = true;                           // no copy's wait has given up
    auto leave = [&]() {
        // the copies in flight land before the CTA's memory goes: a ring has
        // all its slots issued, a resident share none after the first sweep
        if (!m.resident && lane == 0) {
            for (int k = 0; k < m.slots; k++) {
                bool landed = true;
                m.take(0, true, landed);
            }
        }
        __syncwarp();
    };

    // ---- prologue, as k_cn_half's ----
    const bool pred = a.delta != nullptr;
    const bool lin = a.dext != nullptr;
    R *cur = a.q0, *nxt = a.q1;
    double rr0, stop2, rr_last;
    bool converged;
    {
        double v[3] = {0.0, 0.0, 0.0};
        const R *dv0 = lin ? a.dext : a.delta;
        for (int j = warp; j < ns; j += nw) {
            const int row = (sh.s0 + j) * kSlice + lane, beg = sp[j], w = (sp[j + 1] - beg) / kSlice;
            const bool on = row >= rb && row < re;
            const R di = on ? __ldg(a.dinv + row) : R(1), d0 = on && pred ? dv0[row] : R(0);
            R ax = R(0), bx = R(0), ad = R(0);
            mat_slice<R, 1>(m, a, w, true, lane, ok, [&](int c, int k) {
                return Own<R>{a.x[c], __ldg(a.Bval + beg + k * kSlice + lane), pred ? dv0[c] : R(0)};
            }, [&](R av, const Own<R> &t) {
                ax += av * t.p;
                bx += t.q * t.p;
                ad += av * t.d;
            });
            if (on) {
                const R rref = bx - ax;
                const R r = pred ? rref - ad : rref;
                pair_store(cur, row, di * r, R(0));
                own_store(a, row, R(0), R(0), d0);
                v[0] += (double)r * (double)r;
                v[1] += (double)bx * (double)bx;
                v[2] += (double)rref * (double)rref;
            }
        }
        double t[3];
        if (!group_reduce(a.slots, G, ++tag, b0, nb, a.bar_extra, bar, v, t, ok)) { leave(); return; }
        rr0 = t[2];
        stop2 = fmax(a.tol * a.tol * rr0, a.floor_rel * a.floor_rel * t[1]);
        rr_last = t[0];
        converged = t[0] <= stop2;
    }
    int it = 0;
    R al = R(0), be = R(0);
    while (!converged && it < a.maxit) {
        double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        if (m.resident) m.ccol = 0;
        for (int j = warp; j < ns; j += nw) {
            const int row = (sh.s0 + j) * kSlice + lane, w = (sp[j + 1] - sp[j]) / kSlice;
            const bool on = row >= rb && row < re;
            Pair<R> t{R(0), R(0)};
            Own<R> o{R(0), R(0), R(0)};
            R di = R(1);
            if (on) { t = pair_load(cur, row); o = own_load(a, row); di = __ldg(a.dinv + row); }
            R u = R(0);
            mat_slice<R, GU>(m, a, w, false, lane, ok, [&](int c, int) { return pair_z(cur, c, al); },
                             [&](R av, R g) { u += av * g; });
            if (on) sweep_row(a, nxt, row, di, t, o, u, al, be, v);
        }
        double t[7];
        if (!group_reduce(a.slots, G, ++tag, b0, nb, a.bar_extra, bar, v, t, ok)) { leave(); return; }
        { R *sw = cur; cur = nxt; nxt = sw; }
        // the scalars and tests of k_cn_half
        if (t[4] <= stop2) { rr_last = t[4]; converged = true; al = R(0); break; }
        const double alpha = t[1] / t[0], irz = 1.0 / t[1];
        const double rz = t[1] - 2.0 * alpha * t[2] + alpha * alpha * t[3];
        rr_last = t[4] - 2.0 * alpha * t[5] + alpha * alpha * t[6];
        it++;
        al = (R)alpha;
        be = (R)(rz * irz);
        if (!isfinite(rr_last)) break;
        converged = rr_last <= stop2 && stop2 >= 1e-12 * t[4];
    }
    leave();
    cg_finish(a, sh, warp, nw, lane, cur, al, be, converged, tag, it, rr_last, rr0);
}

// ---------------------------------------------------------------------------
// k_cn_one: the solve on one CTA, for meshes whose matrix fits one SM's shared
// memory.  There an iteration needs no other memory: the matrix, the gathered z'
// and the reductions are in shared memory, and a thread keeps the vectors of its
// NR rows in registers: 715 nodes, 4.3 us an iteration to 2.2 in FP64, 3.3 to 2.1
// in FP32.  Two CTA barriers stand in for the grid reduction's
// store, fence and polls.  What is left is a chain of instructions with few warps
// to hide it, so the matrix lies four columns to a lane's load (values, and byte
// offsets into z in 16 bits), its slices padded with zeros to whole groups.
// Same iterates as the other kernels.
__host__ __device__ constexpr int one_cols(long long cols, int ns) {
    return (int)((cols + 3 * (long long)ns + 3) / 4 * 4);       // with the padding, at most
}
template <typename R> __host__ __device__ constexpr long long one_bytes(long long cols, int ns) {
    return kSlice * (ns * (long long)sizeof(R) + one_cols(cols, ns) * (2 + (long long)sizeof(R)));
}
// the four values of a group, from lane's place in it
__device__ __forceinline__ void one_values(const float *g, int lane, float (&v)[4]) {
    const float4 t = reinterpret_cast<const float4 *>(g)[lane];
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void one_values(const double *g, int lane, double (&v)[4]) {
    const double2 t = reinterpret_cast<const double2 *>(g)[lane], u = reinterpret_cast<const double2 *>(g)[32 + lane];
    v[0] = t.x; v[1] = t.y; v[2] = u.x; v[3] = u.y;
}
__device__ __forceinline__ void one_store(float *g, int lane, const float (&v)[4]) {
    reinterpret_cast<float4 *>(g)[lane] = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void one_store(double *g, int lane, const double (&v)[4]) {
    reinterpret_cast<double2 *>(g)[lane] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(g)[32 + lane] = make_double2(v[2], v[3]);
}

// The sums of the CTA's warps, the same bits in every thread, as group_reduce
// forms them, with one barrier: the partials of two calls in turn have their own
// places (buf), so a call's are read while the next one's are written.
template <int NV>
__device__ __forceinline__ void one_reduce(int buf, const double (&vin)[NV], double (&tot)[NV]) {
    __shared__ double sh[2][32][kRedMax], sum[32][kRedMax];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double own = warp_sums(vin);
    if ((lane & 3) == 0) sh[buf][warp][lane >> 2] = own;
    __syncthreads();
    const double t = column_sum(sh[buf], nw);
    if (lane < kRedMax) sum[warp][lane] = t;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < NV; k++) tot[k] = sum[warp][k];
    __syncwarp();
}

template <typename R, int NR>
__global__ void __launch_bounds__(512, 1) k_cn_one(const CGArgs<R> a) {
    extern __shared__ __align__(128) unsigned char cg_sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, ns = a.nslices;
    const CgShare sh = cg_share(a);
    unsigned long long tag = *(volatile unsigned long long *)&a.bar->seq;
    const int first = __ldg(a.slice_ptr), cols = (__ldg(a.slice_ptr + ns) - first) / kSlice;
    // a caller's matrix may be wider than the launch assumed: then it is read
    // from L2 in every sweep
    const bool fits = one_bytes<R>(cols, ns) <= a.smem;
    R *vs = reinterpret_cast<R *>(cg_sm), *zs = vs + (fits ? one_cols(cols, ns) : 0) * kSlice;
    uint2 *is = reinterpret_cast<uint2 *>(zs + ns * kSlice);     // a lane's four offsets
    int beg[NR], grp[NR], w[NR], row[NR];     // entries before the slice, its first group, columns
    bool on[NR];
    R z[NR], q[NR], wv[NR], p[NR], d[NR], di[NR];
#pragma unroll
    for (int k = 0; k < NR; k++) {
        const int s = warp + k * nw;
        row[k] = s * kSlice + lane;
        on[k] = s < ns && row[k] < a.n;
        beg[k] = grp[k] = w[k] = 0;
        if (s < ns) {
            beg[k] = __ldg(a.slice_ptr + s);
            w[k] = (__ldg(a.slice_ptr + s + 1) - beg[k]) / kSlice;
            grp[k] = ((beg[k] - first) / kSlice + 3 * s + 3) / 4;
            zs[row[k]] = on[k] ? a.x[row[k]] : R(0);
        }
        di[k] = on[k] ? __ldg(a.dinv + row[k]) : R(1);
        z[k] = q[k] = wv[k] = p[k] = d[k] = R(0);
    }
    __syncthreads();
    // the row sum of row k, columns in order
    auto row_sum = [&](int k) {
        R u = R(0);
        if (fits) {
            const R *vp = vs + grp[k] * 4 * kSlice;
            const uint2 *ip = is + grp[k] * kSlice + lane;
            const unsigned char *zb = reinterpret_cast<const unsigned char *>(zs);
#pragma unroll (sizeof(R) == 4 ? 4 : 2)
            for (int g = 0; 4 * g < w[k]; g++) {
                const uint2 o = ip[g * kSlice];
                R v[4];
                one_values(vp + g * 4 * kSlice, lane, v);
                const R z0 = *reinterpret_cast<const R *>(zb + (o.x & 0xffffu)), z1 = *reinterpret_cast<const R *>(zb + (o.x >> 16));
                const R z2 = *reinterpret_cast<const R *>(zb + (o.y & 0xffffu)), z3 = *reinterpret_cast<const R *>(zb + (o.y >> 16));
                u += v[0] * z0;
                u += v[1] * z1;
                u += v[2] * z2;
                u += v[3] * z3;
            }
        } else {
            for (int c = 0; c < w[k]; c++) {
                const int e = beg[k] + c * kSlice + lane;
                u += __ldg(a.Aval + e) * zs[__ldg(a.col + e)];
            }
        }
        return u;
    };
    // ---- prologue, as k_cn_half's; the matrix comes in with it ----
    const bool pred = a.delta != nullptr;
    double rr0, stop2, rr_last;
    bool converged;
    {
        double v[3] = {0.0, 0.0, 0.0};
        R ax[NR], bx[NR];
#pragma unroll
        for (int k = 0; k < NR; k++) {
            ax[k] = bx[k] = R(0);
#pragma unroll 2
            for (int c = 0; c < w[k]; c += 4) {
                R av[4], bv[4];
                int ci[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int e = beg[k] + (c + j) * kSlice + lane;
                    const bool in = c + j < w[k];
                    ci[j] = in ? __ldg(a.col + e) : 0;
                    av[j] = in ? __ldg(a.Aval + e) : R(0);
                    bv[j] = in ? __ldg(a.Bval + e) : R(0);
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const R t = zs[ci[j]];
                    if (c + j < w[k]) {
                        ax[k] += av[j] * t;
                        bx[k] += bv[j] * t;
                    }
                }
                if (fits) {
                    const int g = grp[k] + c / 4;
                    constexpr unsigned int S = sizeof(R);
                    one_store(vs + g * 4 * kSlice, lane, av);
                    is[g * kSlice + lane] = make_uint2(S * ci[0] | S * ci[1] << 16, S * ci[2] | S * ci[3] << 16);
                }
            }
        }
        if (pred) {
            const R *dv0 = a.dext ? a.dext : a.delta;
            __syncthreads();
#pragma unroll
            for (int k = 0; k < NR; k++)
                if (on[k]) zs[row[k]] = d[k] = dv0[row[k]];
            __syncthreads();
        }
#pragma unroll
        for (int k = 0; k < NR; k++) {
            const R ad = pred ? row_sum(k) : R(0);
            if (on[k]) {
                const R rref = bx[k] - ax[k], r = pred ? rref - ad : rref;
                z[k] = di[k] * r;
                v[0] += (double)r * (double)r;
                v[1] += (double)bx[k] * (double)bx[k];
                v[2] += (double)rref * (double)rref;
            }
        }
        double t[3];
        if (a.bar_extra) {                    // arrivals that never come (ep_test_hold_barrier)
            if (!group_reduce(a.slots, 1, ++tag, 0, 1, a.bar_extra, a.bar, v, t)) return;
        }
        one_reduce(0, v, t);
        rr0 = t[2];
        stop2 = fmax(a.tol * a.tol * rr0, a.floor_rel * a.floor_rel * t[1]);
        rr_last = t[0];
        converged = t[0] <= stop2;
    }
    int it = 0;
    R al = R(0), be = R(0), diag[NR];
#pragma unroll
    for (int k = 0; k < NR; k++) diag[k] = R(1) / di[k];
    while (!converged && it < a.maxit) {
        double v[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < NR; k++)
            if (on[k]) zs[row[k]] = z[k] = fma(-al, wv[k], z[k]);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NR; k++) {
            const R u = row_sum(k);
            if (on[k]) {
                d[k] = fma(al, p[k], d[k]);
                p[k] = fma(be, p[k], z[k]);
                q[k] = fma(be, q[k], u);
                wv[k] = di[k] * q[k];
                row_sums((double)diag[k], z[k], wv[k], p[k], q[k], v);
            }
        }
        double t[7];
        one_reduce((it & 1) ^ 1, v, t);
        // the scalars and tests of k_cn_half
        if (t[4] <= stop2) { rr_last = t[4]; converged = true; al = R(0); break; }
        const double alpha = t[1] / t[0], irz = 1.0 / t[1];
        const double rz = t[1] - 2.0 * alpha * t[2] + alpha * alpha * t[3];
        rr_last = t[4] - 2.0 * alpha * t[5] + alpha * alpha * t[6];
        it++;
        al = (R)alpha;
        be = (R)(rz * irz);
        if (!isfinite(rr_last)) break;
        converged = rr_last <= stop2 && stop2 >= 1e-12 * t[4];
    }
#pragma unroll
    for (int k = 0; k < NR; k++)
        if (on[k]) finish_row(a, row[k], Pair<R>{z[k], wv[k]}, Own<R>{p[k], q[k], d[k]}, al, be, converged);
    finish_statistics(a, sh, converged, tag, it, rr_last, rr0);
}

// ---------------------------------------------------------------------------
// The same solve by the Chronopoulos-Gear recurrences, whose one reduction an
// iteration gives both scalars as sums of the vectors themselves (k_cn_half's
// next residual is a difference).  With z = dinv r and w = A z,
//   gamma = (r, z), delta = (z, w)                 (one reduction)
//   beta = gamma / gamma_old, alpha = gamma / (delta - beta gamma / alpha_old)
//   p = z + beta p, s = w + beta s, x += alpha p, r -= alpha s
// and the next w = A z is formed in the same pass: each neighbour's new z is
// recomputed from its old r, w, s (read from the other half of r, w, s's
// double buffers), with the owner's explicit fma sequence so both round alike.
// In exact arithmetic the iterates are those of k_cn_half; in floating point
// they differ at the rounding level (an option of the autotuner, not the
// default).
template <typename R>
__device__ __forceinline__ R cg1_snew(R w, R beta, R s) { return fma(beta, s, w); }
template <typename R>
__device__ __forceinline__ R cg1_rnew(R r, R alpha, R snew) { return fma(-alpha, snew, r); }

template <typename R, int NB>
__global__ void __launch_bounds__(NB == 4 ? 768 : 256, NB == 4 ? 2 : 4) k_cn_half_cg1(const CGArgs<R> a) {
    const int lane = threadIdx.x & 31;
    const int G = gridDim.x;
    int inst = 0, b0 = 0, nb = G, rb = 0, re = a.n;
    if (a.ninst > 1) {
        int lo = 0, hi = a.ninst - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.inst_blk[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
        }
        inst = lo;
        b0 = a.inst_blk[inst]; nb = a.inst_blk[inst + 1] - b0;
        rb = a.inst_row[inst]; re = a.inst_row[inst + 1];
    }
    GridBarrier *bar = a.bar + inst;
    const unsigned int nblk = nb + a.bar_extra;
    const int s_lo = rb / kSlice, s_hi = (re + kSlice - 1) / kSlice;
    const int gwarp = s_lo + (((int)blockIdx.x - b0) * (int)blockDim.x + (int)threadIdx.x) / 32;
    const int nwarps = (nb * (int)blockDim.x) >> 5;

    // ---- P1: r0 = B x - A x; p = 0, s_{-1} = 0 ----
    {
        double v[2] = {0.0, 0.0};
        for (int s = gwarp; s < s_hi; s += nwarps) {
            const int row = s * kSlice + lane;
            const int beg = a.slice_ptr[s], w = (a.slice_ptr[s + 1] - beg) / kSlice;
            R ax = R(0), bx = R(0), ad = R(0);
            slice_ab_sums<NB == 4 ? 2 : 4>(a.col, a.Aval, a.Bval, a.x, beg, w, lane, false, [](int) { return R(0); },
                                           ax, bx, ad);
            if (row >= rb && row < re) {
                const R r = bx - ax;
                a.r[row] = r;
                a.p0[row] = R(0);
                a.s1[row] = R(0);
                v[0] += (double)r * (double)r;
                v[1] += (double)bx * (double)bx;
            }
        }
        block_reduce_store<2>(v, a.partial, G);
    }
    if (!grid_sync(bar, nblk)) return;
    double rr0, bb;
    {
        double t[2];
        grid_total<2>(a.partial, G, b0, nb, t);
        rr0 = t[0]; bb = t[1];
    }
    const double stop2 = fmax(a.tol * a.tol * rr0, a.floor_rel * a.floor_rel * bb);
    bool converged = (rr0 <= stop2);
    double rr_last = rr0;
    int it = 0;
    double gamma = 0.0, delta = 0.0;
    // ---- P2: w0 = A z0, gamma0 = (r0, z0), delta0 = (z0, w0) ----
    if (!converged) {
        double v[2] = {0.0, 0.0};
        for (int s = gwarp; s < s_hi; s += nwarps) {
            const int row = s * kSlice + lane;
            const int beg = a.slice_ptr[s], w = (a.slice_ptr[s + 1] - beg) / kSlice;
            const R wv = slice_row_sum<NB>(a.col, a.Aval, beg, w, lane,
                                           [&](int c) { return __ldg(a.dinv + c) * ldcg(a.r + c); });
            if (row >= rb && row < re) {
                const R z = __ldg(a.dinv + row) * a.r[row];
                a.w0[row] = wv;
                v[0] += (double)a.r[row] * (double)z;
                v[1] += (double)z * (double)wv;
            }
        }
        // partial slots: P1 [0, 2G), P2 [9G, 11G), iterations alternate
        // [3G, 6G) and [6G, 9G): consecutive phases never share a slot
        block_reduce_store<2>(v, a.partial + 9 * G, G);
        if (!grid_sync(bar, nblk)) return;
        double t[2];
        grid_total<2>(a.partial + 9 * G, G, b0, nb, t);
        gamma = t[0]; delta = t[1];
    }
    double alpha = (delta > 0.0) ? gamma / delta : 0.0, beta = 0.0;
    if (!(delta > 0.0)) converged = true;       // A z0 = 0: nothing left to solve
    int cur = 0;
    while (!converged && it < a.maxit) {
        const R aR = (R)alpha, bR = (R)beta;
        // the double buffers by selects (no local-memory pointer arrays)
        const R *rc = cur ? a.r1 : a.r, *wc = cur ? a.w1 : a.w0, *sp = cur ? a.s0 : a.s1;
        R *rn = cur ? a.r : a.r1, *wn = cur ? a.w0 : a.w1, *sc = cur ? a.s1 : a.s0;
        double v[3] = {0.0, 0.0, 0.0};
        for (int s = gwarp; s < s_hi; s += nwarps) {
            const int row = s * kSlice + lane;
            const int beg = a.slice_ptr[s], w = (a.slice_ptr[s + 1] - beg) / kSlice;
            // w_{k+1} = A z_{k+1}, z_{k+1} of the neighbours rebuilt from old r, w, s
            const R wv = slice_row_sum<NB>(a.col, a.Aval, beg, w, lane, [&](int c) {
                const R snew = cg1_snew(ldcg(wc + c), bR, ldcg(sp + c));
                return __ldg(a.dinv + c) * cg1_rnew(ldcg(rc + c), aR, snew);
            });
            if (row >= rb && row < re) {
                const R d = __ldg(a.dinv + row);
                const R rk = rc[row];
                const R p = fma(bR, a.p0[row], d * rk);
                const R snew = cg1_snew(wc[row], bR, sp[row]);
                const R rnew = cg1_rnew(rk, aR, snew);
                const R znew = d * rnew;
                a.p0[row] = p;
                sc[row] = snew;
                a.x[row] += aR * p;
                rn[row] = rnew;
                wn[row] = wv;
                v[0] += (double)rnew * (double)znew;
                v[1] += (double)znew * (double)wv;
                v[2] += (double)rnew * (double)rnew;
            }
        }
        block_reduce_store<3>(v, a.partial + 3 * (cur + 1) * G, G);   // alternate slots
        if (!grid_sync(bar, nblk)) return;
        double t[3];
        grid_total<3>(a.partial + 3 * (cur + 1) * G, G, b0, nb, t);
        it++;
        rr_last = t[2];
        converged = (t[2] <= stop2);
        if (!isfinite(t[2])) { converged = false; break; }   // as in k_cn_half
        const double gnew = t[0];
        beta = gnew / gamma;
        const double den = t[1] - beta * gnew / alpha;
        if (!(den > 0.0)) converged = true;        // breakdown at the rounding floor
        alpha = gnew / den;
        gamma = gnew;
        cur = 1 - cur;
    }
    // the solution is in x; r's current buffer is left wherever it is
    if ((int)blockIdx.x == b0 && threadIdx.x == 0) {
        atomicAdd(a.iters_total, (unsigned long long)it);
        atomicMax(a.iters_max, (unsigned int)it);
        if (!converged) atomicAdd(a.fails, 1u);
        if (a.last) {
            a.last[2 * inst] = (double)it;
            a.last[2 * inst + 1] = rr0 > 0.0 ? sqrt(rr_last / rr0) : 0.0;
        }
    }
}

// the kernel of a (gather width, variant) choice and its dynamic shared
// memory; cg_batch kStagedBatch selects k_cn_half's staged form with `depth` units
// in flight per warp (1 .. kStageMaxDepth)
// (set_attr: allow the staged kernel the largest ring any handle can ask
// for -- 256 threads, kStageMaxDepth units -- once, from the planning path,
// never during a stream capture; the attribute only caps the request)
template <typename R>
static int cg_kernel(int block, int batch, int variant, int depth, const void **fn, size_t *smem,
                     bool set_attr, int per_sm = 1) {
    *smem = 0;                 // (k_cn_smem: `depth` is its bytes)
    const bool two = (batch & kTwo) != 0;
    if ((batch & ~kTwo) == kStagedBatch) {
        if (variant != 0) { set_error("the staged CG runs the reference's recurrences only (cg_variant 0)"); return EP_ERR_ARG; }
        if (depth < 1 || depth > kStageMaxDepth) {
            set_error("staged CG: %d units in flight, not 1..%d", depth, kStageMaxDepth);
            return EP_ERR_ARG;
        }
        *fn = two ? (const void *)k_cn_two<R, kStagedBatch> : (const void *)k_cn_half<R, kStagedBatch>;
        *smem = stage_smem_bytes(block, depth, (int)sizeof(R));
        if (set_attr)
            EP_CUDA(cudaFuncSetAttribute(*fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)stage_smem_bytes(256, kStageMaxDepth, (int)sizeof(R))));
        return EP_OK;
    }
    if (two) {
        *fn = batch == kTwo + 8 ? (const void *)k_cn_two<R, 8>
              : batch == kTwo + 16 ? (const void *)k_cn_two<R, 16>
                                   : (const void *)k_cn_two<R, 4>;
        return EP_OK;
    }
    if (batch == kSmemBatch) {
        *fn = (const void *)k_cn_smem<R, 512>;
        *smem = (size_t)depth;
        if constexpr (sizeof(R) == 8) {
            // alone on its SM with fewer threads FP64 has the registers it needs
            // (128 spill); a batch's two CTAs share them
            if (per_sm == 1) *fn = block <= 256 ? (const void *)k_cn_smem<R, 256> : (const void *)k_cn_smem<R, 384>;
        }
        if (set_attr)
            EP_CUDA(cudaFuncSetAttribute(*fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax));
        return EP_OK;
    }
    *fn = variant == 1 ? (batch >= 8 ? (const void *)k_cn_half_cg1<R, 8> : (const void *)k_cn_half_cg1<R, 4>)
          : batch == 8 ? (const void *)k_cn_half<R, 8>
          : batch == 16 ? (const void *)k_cn_half<R, 16>
                        : (const void *)k_cn_half<R, 4, true>;
    return EP_OK;
}

template <typename R>
int cg_max_per_sm(int block, int *per, int batch, int variant, int depth, int per_sm) {
    const void *fn = nullptr;
    size_t smem = 0;
    int rc = cg_kernel<R>(block, batch, variant, depth, &fn, &smem, true, per_sm);
    if (rc) return rc;
    cudaFuncAttributes fa;
    EP_CUDA(cudaFuncGetAttributes(&fa, fn));
    if (block > fa.maxThreadsPerBlock) {
        set_error("CG gather width %d takes at most %d threads per CTA (asked %d)", batch, fa.maxThreadsPerBlock, block);
        return EP_ERR_ARG;
    }
    EP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per, fn, block, smem));
    if (*per < 1) { set_error("CG kernel cannot be resident with %d threads per CTA", block); return EP_ERR_CUDA; }
    return EP_OK;
}

// The launch of a handle that leaves cg_per_sm to the library (0) and keeps
// cg_block 256, cg_batch 4 and cg_variant 0, and of ep_cn_half_step_noalloc.
// No more CTAs than there are slices for, since every CTA takes part in each
// iteration's reduction (measured: CG us a step, two solves, 16-30 iterations):
//   up to 64 slices, where the matrix fits one SM: k_cn_one, whose iterations
//     need no global memory (FP32 / FP64: 280 nodes 33 / 49 us, with the other
//     kernels 49 / 143; 715 nodes 48 / 76 against 74 / 145; 1200 nodes 58 / 101
//     against 92 / 149; 1900 nodes FP32 77 against 92);
//   k_cn_smem where a CTA's share of the matrix stays in shared memory, one CTA
//     per SM: 256 threads up to 8 slices per SM in FP32 and 6 in FP64 (28.6K
//     nodes, FP32: 103 us, 109 with 512 threads, 141 with k_cn_half; 14K FP64:
//     150, 160 with 384, 178 with 256 of 128 registers), beyond it 512 in FP32
//     (214K nodes: 162 us against 195 with 384 and 191 with k_cn_half) and 384
//     in FP64, whose 168 registers hold a slice's gathers without spills (34K:
//     158 us against 199 with 512; 91K: 210 against 260).  FP32 may fill 200 KB
//     with it, FP64 140, whose gathers need the L1 more;
//   k_cn_half with 1024 threads per SM where the matrix no longer does but L2
//     holds it, up to 60 MB in FP32 (263K: 220 us against 270 from the ring;
//     500K: 320 against 374): twice the warps hide L2's latency as well, and
//     nothing is copied; in FP64 up to 27 MB (133K: 281 against 310; 153K 370
//     against 317);
//   k_cn_smem's ring beyond (765K FP32: 630 us against 748; 306K FP64: 540
//     against 710; 562K: 869, 973 with 512 threads), with 120 KB, which leaves
//     the gathers their L1; and k_cn_two for the largest (cg_fit).
// Batches the same with two CTAs per SM, which split the GPU more evenly
// between the instances (24 slabs, 446K nodes FP32: 306 us from k_cn_half, 389
// from the ring); in FP64, whose CTAs want the registers, with one up to a
// quarter as many instances as SMs (CG us a step with one / two: 8 slabs, 155K
// nodes 315 / 309; 24, 446K 625 / 723; 36, 667K 999 / 1031 and 111K 216 / 205;
// beyond, 40 slabs of 123K 287 / 216, 72 of 222K 351 / 304 and of 1.3M 2592 /
// 1901, though small ones still gain: 72 of 36K 119 / 151).
// Any other launch config, and more instances than those CTAs, run k_cn_half, or
// k_cn_two (cg_named_two), with CTAs of `block` threads, as many as fit.
// slices a warp of k_cn_one takes (measured for each, FP32 / FP64, CG us a step:
// 9 slices 33 / 49 with one, 36 / 54 with two; 23 slices 54 / 86, 48 / 76 with
// two, 50 / 82 with three; 38 slices, three 58 / 101, four 66 / 116: fewer warps
// shuffle less in the reductions, up to where the rows' own chains add up)
static int one_rows(int nslices) { return nslices <= 12 ? 1 : nslices <= 32 ? 2 : nslices <= 48 ? 3 : 4; }
template <typename R>
static const void *one_kernel(int nslices) {
    switch (one_rows(nslices)) {
    case 1: return (const void *)k_cn_one<R, 1>;
    case 2: return (const void *)k_cn_one<R, 2>;
    case 3: return (const void *)k_cn_one<R, 3>;
    default: return (const void *)k_cn_one<R, 4>;
    }
}

template <typename R>
int cg_auto_shape(int nslices, long long cols, int ninst, int batch, int variant, int depth, CgShape *out) {
    int dev = 0, nsm = 0, per = 0;
    EP_CUDA(cudaGetDevice(&dev));
    EP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    out->batch = batch;
    out->ring_cols = out->smem = 0;
    if (variant == 0 && (batch & ~kTwo) == 4 && out->block == 256 && ninst <= 2 * nsm) {
        if (ninst == 1 && nslices <= 64 && one_bytes<R>(cols, nslices) <= kOneMax) {
            out->batch = kOneBatch;
            out->block = 32 * div_up(nslices, one_rows(nslices));
            out->grid = out->per_sm = 1;
            out->smem = kOneMax;
            EP_CUDA(cudaFuncSetAttribute(one_kernel<R>(nslices), cudaFuncAttributeMaxDynamicSharedMemorySize, kOneMax));
            return EP_OK;
        }
        out->batch = kSmemBatch;
        // (FP64 batches keep one CTA per SM while an instance has four SMs or more)
        out->per_sm = ninst > 1 && (sizeof(R) == 4 || 4 * ninst > nsm) ? 2 : 1;
        out->block = out->per_sm == 2 || nslices <= (sizeof(R) == 4 ? 8 : 6) * nsm ? 256 : sizeof(R) == 4 ? 512 : 384;
        out->grid = std::min(out->per_sm * nsm, div_up(nslices, out->block / 32) + (ninst > 1 ? ninst : 0));
        return EP_OK;
    }
    int rc = cg_max_per_sm<R>(out->block, &per, batch, variant, depth);
    if (rc) return rc;
    if (ninst > nsm * per && out->block > 128) {
        // more instances than CTAs of this size fit: a warp group each
        out->block = 128;
        if ((rc = cg_max_per_sm<R>(out->block, &per, batch, variant, depth))) return rc;
    }
    // an instance's share of the slices is rounded up to whole CTAs
    out->grid = std::min(nsm * per, div_up(nslices, out->block / 32) + (ninst > 1 ? ninst : 0));
    return EP_OK;
}

template <typename R>
int cg_fit_smem(int ns, long long cols, int nslices, int ninst, int largest, CgShape *out) {
    int per = 0;
    if (!cg_fit<R>(ns, cols, nslices, ninst, largest, out)) {
        if (out->grid) return EP_OK;
        int dev = 0, nsm = 0;
        EP_CUDA(cudaGetDevice(&dev));
        EP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
        const int rc = cg_max_per_sm<R>(out->block, &per, out->batch);
        out->grid = std::min(std::min(per, out->per_sm) * nsm, div_up(nslices, out->block / 32) + (ninst > 1 ? ninst : 0));
        return rc;
    }
    int rc = cg_max_per_sm<R>(out->block, &per, kSmemBatch, 0, out->smem, out->per_sm);
    if (!rc && per < out->per_sm) { set_error("CG kernel: %d CTAs per SM instead of %d", per, out->per_sm); rc = EP_ERR_CUDA; }
    return rc;
}

template <typename R>
int cg_grid_size(int block, int *grid, int per_sm, int batch, int variant, int depth) {
    int dev = 0, nsm = 0, per = 0;
    EP_CUDA(cudaGetDevice(&dev));
    EP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    int rc = cg_max_per_sm<R>(block, &per, batch, variant, depth);
    if (rc) return rc;
    if (per_sm > 0 && per_sm < per) per = per_sm;
    *grid = nsm * per;
    return EP_OK;
}

template <typename R>
int launch_cg(const CGArgs<R> &a, int grid, int block, cudaStream_t s, int batch, int variant) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (batch == kOneBatch) {
        cfg.dynamicSmemBytes = a.smem;
        void *args[] = {const_cast<CGArgs<R> *>(&a)};
        EP_CUDA(cudaLaunchKernelExC(&cfg, one_kernel<R>(a.nslices), args));
    } else if (batch == kSmemBatch) {
        cfg.dynamicSmemBytes = a.smem;
        const void *fn = nullptr;
        size_t smem = 0;
        int rc = cg_kernel<R>(block, batch, variant, a.smem, &fn, &smem, false, a.per_sm);
        if (rc) return rc;
        void *args[] = {const_cast<CGArgs<R> *>(&a)};
        EP_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
    } else if ((batch & kTwo) || batch == kStagedBatch) {
        if ((batch & kTwo) && !a.partial) { set_error("the two-pass CG needs its partial sums"); return EP_ERR_ARG; }
        const void *fn = nullptr;
        size_t smem = 0;
        int rc = cg_kernel<R>(block, batch, variant, a.depth, &fn, &smem, false);
        if (rc) return rc;
        cfg.dynamicSmemBytes = smem;
        void *args[] = {const_cast<CGArgs<R> *>(&a)};
        EP_CUDA(cudaLaunchKernelExC(&cfg, fn, args));
    } else if (variant == 1) {
        if (!a.r1 || !a.w0 || !a.w1 || !a.s0 || !a.s1) { set_error("single-reduction CG needs its vectors"); return EP_ERR_ARG; }
        if (batch >= 8) EP_CUDA(cudaLaunchKernelEx(&cfg, k_cn_half_cg1<R, 8>, a));
        else EP_CUDA(cudaLaunchKernelEx(&cfg, k_cn_half_cg1<R, 4>, a));
    } else if (batch == 8) {
        EP_CUDA(cudaLaunchKernelEx(&cfg, k_cn_half<R, 8>, a));
    } else if (batch == 16) {
        EP_CUDA(cudaLaunchKernelEx(&cfg, k_cn_half<R, 16>, a));
    } else if (grid > kRedFlat) {
        EP_CUDA(cudaLaunchKernelEx(&cfg, k_cn_half<R, 4, true>, a));
    } else {
        EP_CUDA(cudaLaunchKernelEx(&cfg, k_cn_half<R, 4, false>, a));
    }
    return EP_OK;
}

template int launch_cg<float>(const CGArgs<float> &, int, int, cudaStream_t, int, int);
template int launch_cg<double>(const CGArgs<double> &, int, int, cudaStream_t, int, int);
template int cg_auto_shape<float>(int, long long, int, int, int, int, CgShape *);
template int cg_auto_shape<double>(int, long long, int, int, int, int, CgShape *);
template int cg_fit_smem<float>(int, long long, int, int, int, CgShape *);
template int cg_fit_smem<double>(int, long long, int, int, int, CgShape *);
template int cg_grid_size<float>(int, int *, int, int, int, int);
template int cg_grid_size<double>(int, int *, int, int, int, int);
template int cg_max_per_sm<float>(int, int *, int, int, int, int);
template int cg_max_per_sm<double>(int, int *, int, int, int, int);

// ---------------------------------------------------------------------------
// One forward-Euler diffusion sub-step of the explicit scheme
// (EP_ExplicitSolver::Solve, Solvers/EP_ExplicitSolver.cc:54-83):
// out_i = V_i + h (D V)_i / C_L,i with D = -K in the SELL operator.
template <typename R>
__global__ void __launch_bounds__(256) k_explicit(int n, int nslices, const int *__restrict__ slice_ptr,
                                                  const int *__restrict__ col, const R *__restrict__ Dval,
                                                  const R *__restrict__ cl, const R *__restrict__ V, R *out, R h) {
    const int lane = threadIdx.x & 31;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    for (int s = gwarp; s < nslices; s += nwarps) {
        const int row = s * kSlice + lane;
        const int beg = slice_ptr[s], w = (slice_ptr[s + 1] - beg) / kSlice;
        const R d = slice_row_sum<4>(col, Dval, beg, w, lane, [&](int c) { return __ldg(V + c); });
        if (row < n) out[row] = V[row] + h * d / cl[row];
    }
}

template <typename R>
int launch_explicit(int n, int nslices, const int *slice_ptr, const int *col, const R *Dval, const R *cl, R *V,
                    R *tmp, double h, cudaStream_t s) {
    int dev = 0, nsm = 148;
    EP_CUDA(cudaGetDevice(&dev));
    EP_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int grid = std::max(1, std::min(8 * nsm, (nslices + 7) / 8));
    k_explicit<R><<<grid, 256, 0, s>>>(n, nslices, slice_ptr, col, Dval, cl, V, tmp, (R)h);
    EP_CUDA(cudaGetLastError());
    EP_CUDA(cudaMemcpyAsync(V, tmp, sizeof(R) * (size_t)n, cudaMemcpyDeviceToDevice, s));
    return EP_OK;
}

template int launch_explicit<float>(int, int, const int *, const int *, const float *, const float *, float *,
                                     float *, double, cudaStream_t);
template int launch_explicit<double>(int, int, const int *, const int *, const double *, const double *, double *,
                                      double *, double, cudaStream_t);

// ---------------------------------------------------------------------------
// pseudo-ECG: out[f * ne + k] = sum_i W[k * wpitch + i] V[f * n + i] over
// frames f, FP64 accumulation.  A CTA takes a chunk of nodes and FB frames, so
// the weights are read once for FB frames (one launch a frame read them again
// for each, and its 592 partials a lead were added by one thread in series).
// Partials per chunk, added in order by the last CTA of the frame group.
template <int NE> struct EcgFrames { static constexpr int N = NE <= 4 ? 8 : NE <= 8 ? 4 : 2; };

template <typename R, int NE>
__global__ void __launch_bounds__(256) k_ecg(int n, int ne, const R *__restrict__ W, int wpitch,
                                             const R *__restrict__ V, int frames, double *partial,
                                             unsigned int *counter, double *out, unsigned int *slot, int cap) {
    constexpr int FB = EcgFrames<NE>::N;
    const int f0 = blockIdx.y * FB, nf = min(FB, frames - f0);
    double acc[FB][NE];
#pragma unroll
    for (int f = 0; f < FB; f++)
#pragma unroll
        for (int k = 0; k < NE; k++) acc[f][k] = 0.0;
    const R *Vf = V + (size_t)f0 * n;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double w[NE], v[FB];
#pragma unroll
        for (int k = 0; k < NE; k++) w[k] = k < ne ? (double)__ldg(W + (size_t)k * wpitch + i) : 0.0;
#pragma unroll
        for (int f = 0; f < FB; f++) v[f] = f < nf ? (double)__ldg(Vf + (size_t)f * n + i) : 0.0;
#pragma unroll
        for (int f = 0; f < FB; f++)
#pragma unroll
            for (int k = 0; k < NE; k++) acc[f][k] += w[k] * v[f];
    }
    __shared__ double sh[FB * NE][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int f = 0; f < FB; f++)
#pragma unroll
        for (int k = 0; k < NE; k++) {
            if (f >= nf || k >= ne) continue;
            double t = acc[f][k];
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) sh[f * NE + k][warp] = t;
        }
    __syncthreads();
    // partial of (frame, lead) j at part[j * chunks + chunk]
    const int outs = nf * ne, chunks = gridDim.x;
    double *part = partial + (size_t)f0 * ne * chunks;
    if ((int)threadIdx.x < outs) {
        const int f = threadIdx.x / ne, k = threadIdx.x % ne;
        double t = 0.0;
        for (int w = 0; w < 8; w++) t += sh[f * NE + k][w];
        part[(size_t)threadIdx.x * chunks + blockIdx.x] = t;
    }
    __threadfence();
    __syncthreads();
    __shared__ bool last;
    if (threadIdx.x == 0) last = (atomicAdd(counter + blockIdx.y, 1u) == gridDim.x - 1);
    __syncthreads();
    if (last) {
        __threadfence();
        // with a slot counter the sample goes to row *slot of out (the
        // counter lives on the device so that replayed graphs advance it)
        const unsigned int row = slot ? *(volatile unsigned int *)slot : 0u;
        if ((int)row < cap)
            for (int j = warp; j < outs; j += 8) {
                double t = 0.0;
                for (int b = lane; b < chunks; b += 32) t += __ldcg(part + (size_t)j * chunks + b);
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == 0) out[((size_t)row + f0) * ne + j] = t;
            }
        __syncthreads();
        if (threadIdx.x == 0) {
            counter[blockIdx.y] = 0;
            if (slot) *slot = row + 1u;
        }
    }
}

// CTAs over the nodes: four per SM over all frame groups, or 16 nodes a thread
int ecg_chunks(int n, int ne, int frames) {
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int groups = div_up(frames, ecg_frames(ne));
    return std::max(1, std::min(div_up(n, 256), std::max(div_up(4 * nsm, groups), div_up(n, 16 * 256))));
}
int ecg_frames(int ne) { return ne <= 4 ? 8 : ne <= 8 ? 4 : 2; }

template <typename R>
int launch_ecg(int n, int ne, const R *W, int wpitch, const R *V, int frames, double *partial, unsigned int *counter,
               double *out, int chunks, cudaStream_t s, unsigned int *slot, int cap) {
    if (ne <= 0 || frames <= 0) return EP_OK;
    if (ne > 16) { set_error("at most 16 electrodes"); return EP_ERR_ARG; }
    const dim3 grid(chunks, div_up(frames, ecg_frames(ne)));
    const int c = slot ? cap : 1;
    if (ne <= 4) k_ecg<R, 4><<<grid, 256, 0, s>>>(n, ne, W, wpitch, V, frames, partial, counter, out, slot, c);
    else if (ne <= 8) k_ecg<R, 8><<<grid, 256, 0, s>>>(n, ne, W, wpitch, V, frames, partial, counter, out, slot, c);
    else k_ecg<R, 16><<<grid, 256, 0, s>>>(n, ne, W, wpitch, V, frames, partial, counter, out, slot, c);
    EP_CUDA(cudaGetLastError());
    return EP_OK;
}

template int launch_ecg<float>(int, int, const float *, int, const float *, int, double *, unsigned int *, double *, int,
                               cudaStream_t, unsigned int *, int);
template int launch_ecg<double>(int, int, const double *, int, const double *, int, double *, unsigned int *, double *,
                                int, cudaStream_t, unsigned int *, int);

__global__ void k_step_inc(long long *step) { *step += 1; }
void launch_step_inc(long long *step, cudaStream_t s) { k_step_inc<<<1, 1, 0, s>>>(step); }

}  // namespace ep

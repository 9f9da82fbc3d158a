/* pcg_common.cuh — device pieces shared by the solver kernels (internal). */
#ifndef GSLAM_PCG_COMMON_CUH
#define GSLAM_PCG_COMMON_CUH

#include <cuda_runtime.h>
#include <stdint.h>

#include "gslam.h"
#include "kernels.cuh"

/* largest dynamic shared memory a solver's CTA asks for (sm_100: 227 KB per block with the
 * static part): the cluster solver's, and the grid-wide ones', whose reductions keep up to
 * 5 KB of static shared memory */
#define GSLAM_RES_SMEM_MAX (225 * 1024)
#define GSLAM_GRID_SMEM_MAX (222 * 1024)

__device__ __forceinline__ unsigned ld_relaxed_u32(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned atom_add_release_u32(unsigned *p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

__device__ __forceinline__ int ld_relaxed_s32(const int *p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

/*
 * Grid barrier on a monotonic arrival counter: barrier number `epoch` (1, 2, ...)
 * is complete when the counter reaches epoch * gridDim.x. One release atomic per
 * CTA (it orders the CTA's prior writes, made visible to thread 0 by a CTA
 * barrier before it), then polling: each poll reads the counter and the abort flag
 * with relaxed loads that are in flight together (one L2 round trip per poll), and
 * a fence.acq_rel after the counter is seen complete gives the acquire side. The
 * counter is zeroed before every launch, so 2^32 / gridDim.x barriers fit in one
 * solve. grid_barrier_t0 is thread 0's part alone (the caller has already made the
 * CTA's writes visible to thread 0 and publishes *s_ok after it); grid_barrier is
 * the whole-CTA form. Both report false when the solve must be abandoned (this wait
 * ran out of time, or another CTA's did).
 */
__device__ __forceinline__ void grid_barrier_t0(GridSync *gs, unsigned epoch, long long spin_limit, int *s_ok) {
    int ok = 1;
    const unsigned target = epoch * gridDim.x;
    const unsigned arrived = atom_add_release_u32(&gs->count, 1u) + 1u;
    if (arrived < target) {
        const long long t0 = clock64();
        while (true) {
            const unsigned c = ld_relaxed_u32(&gs->count);
            const int ab = ld_relaxed_s32(&gs->abort);
            if (c >= target) break;
            if (ab) { ok = 0; break; }
            if (clock64() - t0 > spin_limit) {
                atomicExch(&gs->abort, 1);
                ok = 0;
                break;
            }
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
    }
    *s_ok = ok;
}

__device__ __forceinline__ bool grid_barrier(GridSync *gs, unsigned epoch, long long spin_limit,
                                             int *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0) grid_barrier_t0(gs, epoch, spin_limit, s_ok);
    __syncthreads();
    return *s_ok != 0;
}

/*
 * The solve's status record (PcgResult). The host zeroes it before every launch and
 * the kernel only ever RAISES `timeout`: a CTA that gave up at a barrier has already
 * arrived there, so the other CTAs can complete that barrier and finish normally while
 * its rows of x stay behind. Block 0 must then not report success, whichever of the two
 * writes lands last.
 *   res_mark_timeout: any CTA that gave up (or saw another CTA give up);
 *   res_finish:       block 0, thread 0, at the end of a solve its own CTA completed:
 *                     counts and norms, then the reason, or a timeout when any CTA has
 *                     raised the abort flag by then (one that gives up later raises
 *                     `timeout` itself).
 */
__device__ __forceinline__ void res_mark_timeout(PcgResult *res) {
    atomicOr(&res->timeout, 1);
    atomicExch(&res->reason, GSLAM_STOP_TIMEOUT);
}

__device__ __forceinline__ void res_finish(PcgResult *res, const GridSync *gs, int iterations, int reason,
                                           int refinements, double rnorm, double bnorm) {
    res->iterations = iterations;
    res->refinements = refinements;
    res->rnorm = rnorm;
    res->bnorm = bnorm;
    res->reason = reason;
    if (ld_relaxed_s32(&gs->abort)) res_mark_timeout(res);
}

/*
 * Deterministic all-reduce of NV (<= 4) doubles across the grid, in pieces so that
 * a caller can issue loads of data the other CTAs published before the barrier
 * while the partials are summed, and can derive scalars from the totals in one
 * thread instead of all of them:
 *   grid_reduce_arrive:  block sum of each thread's v[] (warp shuffles, then warp 0
 *                        over the warps), one partial per CTA, grid barrier
 *                        (false: the solve must be abandoned);
 *   grid_reduce_sum:     warp i < NV sums the CTAs' partials of value i into
 *                        s_bc[i] (a lane's loads all in flight together, a fixed
 *                        order: lane-strided, then a shuffle tree), then a
 *                        barrier among those NV warps, so thread 0 sees every total;
 *   grid_reduce_collect: grid_reduce_sum, CTA barrier, v[] = the totals everywhere.
 * Two partial buffers alternate: a CTA can be at most one reduction ahead of the
 * slowest reader, so it never overwrites partials still being summed.
 */
#define GSLAM_SUM_UNROLL 5 /* partial loads per lane issued together (grids up to 160 CTAs) */

template <int NV, int BS>
__device__ __forceinline__ bool grid_reduce_arrive(const double (&v)[NV], double *partials_base, int &epoch,
                                                   GridSync *gs, long long spin_limit,
                                                   double (*s_red)[BS / 32], int *s_ok) {
    static_assert(NV <= 4 && BS / 32 <= 32, "reduction shape");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *partials = partials_base + (epoch & 1) * 4 * gridDim.x;
    epoch++;                                   /* this reduction's barrier number */
#pragma unroll
    for (int i = 0; i < NV; i++) {
        double a = v[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a = a + __shfl_down_sync(0xffffffffu, a, o);
        if (lane == 0) s_red[i][warp] = a;
    }
    __syncthreads();
    if (warp == 0) {
        /* warp 0 sums every value's per-warp partials (the trees interleave), and
         * its lane 0 stores them and arrives: no second CTA barrier before the
         * arrival, since the one above already ordered every thread's writes */
        double a[NV];
#pragma unroll
        for (int i = 0; i < NV; i++) a[i] = lane < BS / 32 ? s_red[i][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int i = 0; i < NV; i++) a[i] = a[i] + __shfl_down_sync(0xffffffffu, a[i], o);
        }
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < NV; i++) partials[i * gridDim.x + blockIdx.x] = a[i];
            grid_barrier_t0(gs, (unsigned)epoch, spin_limit, s_ok);
        }
    }
    __syncthreads();
    return *s_ok != 0;
}

template <int NV>
__device__ __forceinline__ void grid_reduce_sum(const double *partials_base, int epoch, double *s_bc) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp >= NV) return;
    const int G = (int)gridDim.x;
    const double *pp = partials_base + ((epoch - 1) & 1) * 4 * G + warp * G;
    double t[GSLAM_SUM_UNROLL];
#pragma unroll
    for (int u = 0; u < GSLAM_SUM_UNROLL; u++) {
        const int c = lane + 32 * u;
        t[u] = c < G ? __ldcg(pp + c) : 0.0;
    }
    double s = t[0];
#pragma unroll
    for (int u = 1; u < GSLAM_SUM_UNROLL; u++) s = s + t[u];
    for (int c = lane + 32 * GSLAM_SUM_UNROLL; c < G; c += 32) s = s + __ldcg(pp + c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) s_bc[warp] = s;
    if (NV > 1) asm volatile("bar.sync 1, %0;" ::"r"(NV * 32) : "memory");
}

template <int NV, int BS>
__device__ __forceinline__ void grid_reduce_collect(double (&v)[NV], const double *partials_base, int epoch,
                                                    double *s_bc) {
    grid_reduce_sum<NV>(partials_base, epoch, s_bc);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; i++) v[i] = s_bc[i];
}

template <int NV, int BS>
__device__ __forceinline__ bool grid_allreduce(double (&v)[NV], double *partials_base, int &epoch,
                                               GridSync *gs, long long spin_limit,
                                               double (*s_red)[BS / 32], double *s_bc, int *s_ok) {
    if (!grid_reduce_arrive<NV, BS>(v, partials_base, epoch, gs, spin_limit, s_red, s_ok)) return false;
    grid_reduce_collect<NV, BS>(v, partials_base, epoch, s_bc);
    return true;
}

/* grid_allreduce of R values per thread: the warp's rows are slices warp and warp + BS / 32,
 * and the CTA's tree runs over its slices (the same sums as one row per thread) */
template <int NV, int R, int BS>
__device__ __forceinline__ bool grid_allreduce_rows(const double (&v)[NV][R], double (&tot)[NV], double *partials_base,
                                                    int &epoch, GridSync *gs, long long spin_limit, double (*s_red)[32],
                                                    double *s_bc, int *s_ok) {
    static_assert(NV <= 4 && R * BS / 32 <= 32, "reduction shape");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *partials = partials_base + (epoch & 1) * 4 * gridDim.x;
    epoch++;
#pragma unroll
    for (int i = 0; i < NV; i++)
#pragma unroll
        for (int j = 0; j < R; j++) {
            double a = v[i][j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a = a + __shfl_down_sync(0xffffffffu, a, o);
            if (lane == 0) s_red[i][warp + j * (BS / 32)] = a;
        }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < NV; i++) {
            double a = lane < R * BS / 32 ? s_red[i][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a = a + __shfl_down_sync(0xffffffffu, a, o);
            if (lane == 0) partials[i * gridDim.x + blockIdx.x] = a;
        }
        if (lane == 0) grid_barrier_t0(gs, (unsigned)epoch, spin_limit, s_ok);
    }
    __syncthreads();
    if (!*s_ok) return false;
    grid_reduce_collect<NV, BS>(tot, partials_base, epoch, s_bc);
    return true;
}

/*
 * The same all-reduce without a barrier counter and without fences. Every value travels with
 * its reduction's number: 16 bytes holding the two halves of a double, each beside the
 * number, written by one 128-bit exchange and polled with 128-bit loads, so a reader that
 * sees the number has the data, and one trip through L2 replaces the counter's three (the
 * release that waits for the partials, the counter, the partials). 148 CTAs x 768 threads,
 * two doubles: 2.40 us with grid_reduce_*, 1.41 with this (one double 1.27; x 384 threads
 * 1.25). Plain stores instead of the exchange, or a mailbox per reader, take 2.1 to 4.6 us:
 * many readers of a line slow the writes to it. That also holds for readers that poll
 * before the data can be there (1.69 us when they poll at once), so the first poll waits
 * TAG_DELAY cycles after the CTA's own value left: the trip's length and part of the CTAs'
 * skew. Resident FP64 solver, us per iteration at 20,000 / 50,000 / 100,000 poses: 600 cycles
 * 3.54 / 4.43 / 5.94, 680 3.49 / 4.34 / 5.95, 750 3.50 / 4.28 / 5.97, 820 3.53 / 4.27 / 6.02 (without
 * a wait 0.6 to 0.7 more than with 700, with 1000 0.1 to 0.3 more, in an earlier form of the
 * solver). Later polls follow at once (a gap of 150 cycles between them costs 0.1 us).
 *
 * The slots are zeroed before every launch; number 1 is the first reduction. Two buffers
 * alternate: a CTA writes number n + 2 only after it has read every CTA's n + 1, which each
 * of them sent after it had read every n.
 *
 * Sums are those of grid_reduce_*, bit for bit: the warps' tree, then the CTAs lane-strided,
 * then the tree over the lanes.
 */
#define TAG_DELAY 750
#define TAG_VALUES 4 /* values of one reduction */

struct TagWord {
    unsigned long long a, b;
};

__device__ __forceinline__ void tag_exch(TagWord *p, double v, unsigned tag) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
    const unsigned long long a = (bits & 0xffffffffull) | t, b = (bits >> 32) | t;
    asm volatile("{\n .reg .b128 q, r;\n mov.b128 q, {%1, %2};\n atom.relaxed.gpu.global.exch.b128 r, [%0], q;\n}\n" ::"l"(p),
                 "l"(a), "l"(b)
                 : "memory");
}
__device__ __forceinline__ void tag_store(TagWord *p, unsigned long long a, unsigned long long b) {
    asm volatile("{\n .reg .b128 q;\n mov.b128 q, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], q;\n}\n" ::"l"(p), "l"(a), "l"(b)
                 : "memory");
}
__device__ __forceinline__ TagWord tag_load(const TagWord *p) {
    TagWord r;
    asm volatile("{\n .reg .b128 q;\n ld.relaxed.gpu.global.b128 q, [%2];\n mov.b128 {%0, %1}, q;\n}\n"
                 : "=l"(r.a), "=l"(r.b)
                 : "l"(p)
                 : "memory");
    return r;
}

/* whether a poll that has failed `n` times must be given up: this wait's time is over (then
 * every other wait's is too), or another wait gave up */
__device__ __forceinline__ bool tag_give_up(GridSync *gs, int n, long long t0, long long limit) {
    if ((n & 15) != 15) return false;
    if (ld_relaxed_s32(&gs->abort)) return true;
    if (clock64() - t0 <= limit) return false;
    atomicExch(&gs->abort, 1);
    return true;
}

/* The warp's sums of N values at once, each in the order of the butterfly 16, 8, 4, 2, 1: at
 * every step a lane keeps one of two values and sends the other, so N = 2 takes 6 shuffles, not
 * 10, N = 4 takes 8, not 20. Value v's sum ends on the lane whose five bits are v's, reversed:
 * the lane with warp_sums_value(lane) == v. With sum_partials below, 50,000 poses: 4.47 -> 4.25
 * us per iteration in FP64, 3.75 -> 3.58 with one reduction, 2.93 -> 2.67 mixed; 100,000 poses
 * 6.18 -> 5.95, 6.22 -> 6.13, 4.45 -> 4.27. */
__device__ __forceinline__ int warp_sums_value(int lane) { return (int)(__brev((unsigned)lane) >> 27); }
template <int N>
__device__ __forceinline__ double warp_sums(double (&a)[N]) {
    const int lane = threadIdx.x & 31;
    int n = N;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int i = 0; 2 * i < N; i++) {
            if (2 * i + 1 < n) {
                const double keep = lane & o ? a[2 * i + 1 < N ? 2 * i + 1 : 0] : a[2 * i];
                const double send = lane & o ? a[2 * i] : a[2 * i + 1 < N ? 2 * i + 1 : 0];
                a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            } else if (2 * i < n) {
                a[i] = a[2 * i] + __shfl_xor_sync(0xffffffffu, a[2 * i], o);
            }
        }
        n = (n + 1) / 2;
    }
    return a[0];
}

/* The sum of M <= 32 partials that every lane can read, on every lane, in the same order: a
 * lane adds every second (M <= 16) or fourth one in registers, one or two shuffles join them. */
template <int M>
__device__ __forceinline__ double sum_partials(const double *v) {
    constexpr int S = M <= 16 ? 2 : 4;
    const int h = threadIdx.x & (S - 1);
    double b[8];
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = S * i + h < M ? v[S * i + h] : 0.0;
    double t = ((b[0] + b[4]) + (b[2] + b[6])) + ((b[1] + b[5]) + (b[3] + b[7]));
    if (S == 4) t = t + __shfl_xor_sync(0xffffffffu, t, 2);
    return t + __shfl_xor_sync(0xffffffffu, t, 1);
}

/* sums of v[][] over the CTA and their way to the slots: by warps 0 .. NV - 1, one value
 * each, after a CTA barrier. v[i][j]: value i of the thread's j-th row; the warp's rows are
 * slices warp and warp + BS / 32, and the CTA's tree runs over its slices. tag: the
 * reduction's number. */
template <int NV, int R, int BS>
__device__ __forceinline__ void tag_reduce_send(const double (&v)[NV][R], TagWord *slots, unsigned tag,
                                                double (*s_red)[32]) {
    static_assert(NV <= TAG_VALUES && R * BS / 32 <= 32, "reduction shape");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double a[NV * R];
#pragma unroll
    for (int i = 0; i < NV; i++)
#pragma unroll
        for (int j = 0; j < R; j++) a[i * R + j] = v[i][j];
    const double w = warp_sums<NV * R>(a);
    const int k = warp_sums_value(lane);
    if (k < NV * R) s_red[k / R][warp + k % R * (BS / 32)] = w;
    __syncthreads();
    if (warp < NV) {
        const double t = sum_partials<R * BS / 32>(s_red[warp]);
        if (lane == 0) tag_exch(slots + ((tag & 1) * TAG_VALUES + warp) * gridDim.x + blockIdx.x, t, tag);
    }
}

/* the totals into s_bc[], for thread 0 (and whoever passes a CTA barrier after it); *s_ok = 0
 * when a wait gave up. Every slot is polled by a thread of its own, into s_slot, and then one
 * warp per value adds them: by the first TAG_WARPS * NV warps, which leave the others to the
 * caller, where the CTA has that many (call it with all threads), else by all. (One warp per
 * value with five slots a lane needs 30 registers in every thread of the kernel: 400 bytes of
 * spills in a 768-thread CTA.) A grid has at most TAG_LANES CTAs. */
#define TAG_WARPS 5
#define TAG_LANES (32 * TAG_WARPS)

template <int NV, int BS>
__device__ __forceinline__ void tag_reduce_sum(const TagWord *slots, unsigned tag, GridSync *gs, long long spin_limit,
                                               double (*s_slot)[TAG_LANES], double *s_bc, int *s_ok) {
    constexpr bool SOME = TAG_WARPS * NV <= BS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (SOME && warp >= TAG_WARPS * NV) return;
    const int G = (int)gridDim.x;
    const TagWord *p = slots + (tag & 1) * TAG_VALUES * G;
    const long long t0 = clock64();
    while (clock64() - t0 < TAG_DELAY) {}
    for (int c = threadIdx.x; c < NV * TAG_LANES; c += BS) {
        const int v = c / TAG_LANES, l = c - v * TAG_LANES;
        double d = 0.0;
        if (l < G) {
            TagWord w = tag_load(p + v * G + l);
            for (int n = 0; (unsigned)(w.a >> 32) != tag || (unsigned)(w.b >> 32) != tag; n++) {
                if (tag_give_up(gs, n, t0, spin_limit)) { *s_ok = 0; break; }
                w = tag_load(p + v * G + l);
            }
            d = __longlong_as_double((long long)((w.a & 0xffffffffull) | w.b << 32));
        }
        s_slot[v][l] = d;
    }
    if (SOME) asm volatile("bar.sync 1, %0;" ::"r"(NV * TAG_LANES) : "memory");
    else __syncthreads();
    if (warp < NV) {
        double t = s_slot[warp][lane];
#pragma unroll
        for (int u = 1; u < TAG_WARPS; u++) t = t + s_slot[warp][lane + 32 * u];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = t + __shfl_down_sync(0xffffffffu, t, o);
        if (lane == 0) s_bc[warp] = t;
        if (NV > 1) asm volatile("bar.sync 2, %0;" ::"r"(NV * 32) : "memory");
    }
}

struct V3 { double a, b, c; };

__device__ __forceinline__ V3 ld3(const double *v4, int row) {
    const double2 lo = *reinterpret_cast<const double2 *>(v4 + 4 * (size_t)row);
    const double hi = v4[4 * (size_t)row + 2];
    return V3{ lo.x, lo.y, hi };
}

/* L2-only loads for data other CTAs write during the kernel (z, p, partials): never
 * served from this SM's L1, so correctness does not depend on L1 invalidation. */
__device__ __forceinline__ V3 ldcg3(const double *v4, int row) {
    const double2 lo = __ldcg(reinterpret_cast<const double2 *>(v4 + 4 * (size_t)row));
    const double hi = __ldcg(v4 + 4 * (size_t)row + 2);
    return V3{ lo.x, lo.y, hi };
}

/* read-only (non-coherent path) variant for data no CTA writes during the kernel */
__device__ __forceinline__ V3 ldg3(const double *v4, int row) {
    const double2 lo = __ldg(reinterpret_cast<const double2 *>(v4 + 4 * (size_t)row));
    const double hi = __ldg(v4 + 4 * (size_t)row + 2);
    return V3{ lo.x, lo.y, hi };
}

__device__ __forceinline__ void st3(double *v4, int row, V3 v) {
    *reinterpret_cast<double2 *>(v4 + 4 * (size_t)row) = make_double2(v.a, v.b);
    v4[4 * (size_t)row + 2] = v.c;
}

/* a row of three doubles published for the CTAs that read it, with the number of the
 * iteration it belongs to in both halves (32 bytes: a double, the next one's low word and
 * the number; its high word and the number, a double) */
__device__ __forceinline__ void tag_row_store(double *v4, int row, V3 v, unsigned tag) {
    TagWord *p = reinterpret_cast<TagWord *>(v4 + 4 * (size_t)row);
    const unsigned long long b = (unsigned long long)__double_as_longlong(v.b), t = (unsigned long long)tag << 32;
    tag_store(p, (unsigned long long)__double_as_longlong(v.a), (b & 0xffffffffull) | t);
    tag_store(p + 1, (b >> 32) | t, (unsigned long long)__double_as_longlong(v.c));
}
/* reads such a row, waiting for the number; false (the row unknown) when the wait gave up */
__device__ __forceinline__ bool tag_row_load(const double *v4, int row, unsigned tag, GridSync *gs, long long spin_limit,
                                             V3 *v) {
    const TagWord *p = reinterpret_cast<const TagWord *>(v4 + 4 * (size_t)row);
    const long long t0 = clock64();
    for (int n = 0;; n++) {
        const TagWord a = tag_load(p), b = tag_load(p + 1);
        if ((unsigned)(a.b >> 32) == tag && (unsigned)(b.a >> 32) == tag) {
            *v = V3{ __longlong_as_double((long long)a.a),
                     __longlong_as_double((long long)((a.b & 0xffffffffull) | b.a << 32)), __longlong_as_double((long long)b.b) };
            return true;
        }
        if (tag_give_up(gs, n, t0, spin_limit)) return false;
    }
}

/* the smallest number whose rounded square root is not below tol, so that
 * rr < square_limit(tol) decides as sqrt(rr) < tol does (sqrt is monotonic and correctly
 * rounded) without a square root on the critical path; no root is below a tol of 0 or less */
__device__ __forceinline__ double square_limit(double tol) {
    if (tol <= 0.0) return 0.0;
    double y = tol * tol;
    for (int i = 0; i < 8 && sqrt(y) < tol; i++) y = __longlong_as_double(__double_as_longlong(y) + 1);
    for (int i = 0; i < 8 && y > 0.0 && sqrt(__longlong_as_double(__double_as_longlong(y) - 1)) >= tol; i++)
        y = __longlong_as_double(__double_as_longlong(y) - 1);
    return y;
}

/* p_new = z + beta * p_old exactly as MatrixOps.c:382 (first iteration: p = z). */
__device__ __forceinline__ V3 p_of(const double *z4, const double *pold4, int row, double beta,
                                   bool first) {
    V3 z = ldcg3(z4, row);
    if (first) return z;
    V3 p = ldcg3(pold4, row);
    return V3{ z.a + beta * p.a, z.b + beta * p.b, z.c + beta * p.c };
}

/* z = D^-1 r: z_i = ((0 + d_i0 r0) + d_i1 r1) + d_i2 r2 (MatrixOps.c:369-377). */
__device__ __forceinline__ V3 apply_dinv(const double *dinv, int row, V3 r) {
    const double *d = dinv + 288 * (size_t)(row >> 5) + (row & 31);
    double z0 = 0.0, z1 = 0.0, z2 = 0.0;
    z0 = z0 + __ldg(d + 0) * r.a;   z0 = z0 + __ldg(d + 32) * r.b;  z0 = z0 + __ldg(d + 64) * r.c;
    z1 = z1 + __ldg(d + 96) * r.a;  z1 = z1 + __ldg(d + 128) * r.b; z1 = z1 + __ldg(d + 160) * r.c;
    z2 = z2 + __ldg(d + 192) * r.a; z2 = z2 + __ldg(d + 224) * r.b; z2 = z2 + __ldg(d + 256) * r.c;
    return V3{ z0, z1, z2 };
}

/* q += block (3x3, slot layout at v) * p, each scalar row in column order. */
__device__ __forceinline__ void blk_acc(const double *v, V3 p, double &q0, double &q1, double &q2) {
    q0 = q0 + __ldg(v + 0) * p.a;   q0 = q0 + __ldg(v + 32) * p.b;  q0 = q0 + __ldg(v + 64) * p.c;
    q1 = q1 + __ldg(v + 96) * p.a;  q1 = q1 + __ldg(v + 128) * p.b; q1 = q1 + __ldg(v + 160) * p.c;
    q2 = q2 + __ldg(v + 192) * p.a; q2 = q2 + __ldg(v + 224) * p.b; q2 = q2 + __ldg(v + 256) * p.c;
}

/* Same as blk_acc for values that may live in shared or global memory. */
__device__ __forceinline__ void blk_acc_any(const double *v, V3 p, double &q0, double &q1, double &q2) {
    q0 = q0 + v[0] * p.a;   q0 = q0 + v[32] * p.b;  q0 = q0 + v[64] * p.c;
    q1 = q1 + v[96] * p.a;  q1 = q1 + v[128] * p.b; q1 = q1 + v[160] * p.c;
    q2 = q2 + v[192] * p.a; q2 = q2 + v[224] * p.b; q2 = q2 + v[256] * p.c;
}

/*
 * One row of q = A p with p formed on the fly from z and the previous p. Two
 * blocks per step so both columns' gathers are in flight together; blocks are
 * still added in ascending column order.
 */
__device__ __forceinline__ V3 spmv_row(const double *vb, const int *cb, int len, const double *z4,
                                       const double *pold, double beta, bool first) {
    double q0 = 0.0, q1 = 0.0, q2 = 0.0;
    int j = 0;
    for (; j + 1 < len; j += 2) {
        const int c0 = __ldg(cb + 32 * j), c1 = __ldg(cb + 32 * (j + 1));
        const V3 p0 = p_of(z4, pold, c0, beta, first);
        const V3 p1 = p_of(z4, pold, c1, beta, first);
        blk_acc(vb + 288 * j, p0, q0, q1, q2);
        blk_acc(vb + 288 * (j + 1), p1, q0, q1, q2);
    }
    if (j < len) {
        const int c0 = __ldg(cb + 32 * j);
        blk_acc(vb + 288 * j, p_of(z4, pold, c0, beta, first), q0, q1, q2);
    }
    return V3{ q0, q1, q2 };
}

#endif

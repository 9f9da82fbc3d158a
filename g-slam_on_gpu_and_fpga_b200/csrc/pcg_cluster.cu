/*
 * pcg_cluster.cu — block-Jacobi PCG of a whole graph inside one thread-block cluster
 * (reference algorithm: src/cpu_pcg_fp64/MatrixOps.c:281-391).
 *
 * The grid-wide solvers spend most of an iteration in their two grid reductions, each of
 * several L2 round trips: with 148 CTAs of 768 threads one all-reduce of two doubles takes
 * 2.4 us, whatever the graph's size. Inside one cluster the same reduction through
 * distributed shared memory takes 0.66 us (16 CTAs x 256 threads) to 0.87 us (16 x 768),
 * and a cluster's shared memory (16 x 227 KB) holds the matrix of a graph of about 10,000
 * poses. So a graph that fits is solved by one cluster of 1 to 16 CTAs, and a batch by one
 * cluster per graph, as many at a time as the GPU holds, unless the grid-wide solvers are
 * estimated to be faster (long rows, rows read by many CTAs: gslam_cluster_us).
 *
 * Layout: CTA r of a graph's cluster owns a contiguous range of its slices (balanced by
 * slot count), one thread per block row (two above 20 slices per CTA). Values (as far as they
 * fit; every slice leaves out its last block positions, so that no warp is much slower than
 * the others: 8.2 us per iteration at 16,000 poses against 9.5 with whole slices left out),
 * CTA-local column indices and p of own and halo rows are in shared memory; x, r, z, p, q
 * and, with one row per thread, the row's D^-1 are in registers. Nothing but the values that
 * do not fit (and D^-1 of two rows) is read from L2 during the solve.
 *
 * Exchange: warp 0 adds its CTA's partials and stores the sum into every CTA of the cluster
 * (st.async: the data and the count on the receiver's mbarrier in one message, no fence and
 * no polling of global memory); each owner stores z of a row that other CTAs read into
 * their halo arrays the same way, while the sums travel. A CTA's mbarrier completes when
 * all sums, and the halo's z, are there: one one-way trip per reduction. Warp 0 then adds
 * the sums and one thread advances the scalars. (Every warp storing its own slice's sum
 * into every CTA saves the step through warp 0, but the 320 messages per CTA and reduction
 * of a 16 x 640 cluster take longer: in the first form of this kernel 6.6 us per iteration at
 * 10,000 poses against 4.8, and 5.2 against 4.0 at 7,120, which takes 3.0 now.)
 *
 * The two barriers' phases alternate (p.q, then r.r and r.z), and a CTA sends its sums of
 * phase n + 1 only after it has received every sum of phase n, so one buffer and one
 * mbarrier per kind are enough: no CTA can overwrite sums, or a halo's z, that another one
 * still reads (that one's sums of the phase in between come after those reads).
 *
 * Summation orders. Each scalar row of q adds its blocks in ascending original column
 * order with separate multiply and add, as everywhere. Dot products are summed per slice,
 * then per CTA, then over the CTAs. A single graph's cluster of one CTA sums exactly as the
 * grid-wide solver (pcg_resident.cu) does: per slice, per CTA of that solver's partition
 * (vcta_slice; the same tree over its warps), then over its CTAs, so both give the same
 * bits: the solves of such small graphs can go on past convergence, where rounding alone
 * decides the iterates.
 *
 * T = float is the inner solve of the mixed batch (FP32 values and vectors, FP64 D^-1 and
 * dot products), with batch.cu's arithmetic.
 *
 * Waits are bounded: a wait that runs out marks the solve as timed out and the CTA leaves
 * through the final cluster barrier, and a little after it (no CTA exits while another's
 * store into its shared memory may be on its way).
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "cluster_common.cuh"
#include "gslam.h"
#include "kernels.cuh"
#include "pcg_common.cuh"
#include "tma_bulk.cuh"

template <typename T> struct C3 { T a, b, c; };

__device__ __forceinline__ C3<double> cl_ld_row(const double *v4, int row) {
    const V3 v = ldg3(v4, row);
    return { v.a, v.b, v.c };
}
__device__ __forceinline__ C3<float> cl_ld_row(const float *v4, int row) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(v4 + 4 * (size_t)row));
    return { v.x, v.y, v.z };
}
__device__ __forceinline__ void cl_st_row(double *v4, int row, C3<double> v) { st3(v4, row, V3{ v.a, v.b, v.c }); }
__device__ __forceinline__ void cl_st_row(float *v4, int row, C3<float> v) {
    *reinterpret_cast<float4 *>(v4 + 4 * (size_t)row) = make_float4(v.a, v.b, v.c, 0.f);
}

/* z of halo slot h: FP64 as 16 + 8 bytes in two arrays, FP32 as one float4 */
__device__ __forceinline__ void cl_send_z(unsigned zh, unsigned zh2, unsigned rank, int h, C3<double> z, unsigned bar) {
    const unsigned rb = cl_mapa(bar, rank);
    cl_st_async2(cl_mapa(zh + 16 * h, rank), z.a, z.b, rb);
    cl_st_async(cl_mapa(zh2 + 8 * h, rank), z.c, rb);
}
__device__ __forceinline__ void cl_send_z(unsigned zh, unsigned, unsigned rank, int h, C3<float> z, unsigned bar) {
    cl_st_async4(cl_mapa(zh + 16 * h, rank), z.a, z.b, z.c, cl_mapa(bar, rank));
}
template <typename T>
__device__ __forceinline__ C3<T> cl_halo_z(const unsigned char *zh, const unsigned char *zh2, int h);
template <> __device__ __forceinline__ C3<double> cl_halo_z<double>(const unsigned char *zh, const unsigned char *zh2, int h) {
    const double2 ab = *reinterpret_cast<const double2 *>(zh + 16 * h);
    return { ab.x, ab.y, *reinterpret_cast<const double *>(zh2 + 8 * h) };
}
template <> __device__ __forceinline__ C3<float> cl_halo_z<float>(const unsigned char *zh, const unsigned char *, int h) {
    const float4 v = *reinterpret_cast<const float4 *>(zh + 16 * h);
    return { v.x, v.y, v.z };
}

/* z = D^-1 r in FP64 from the nine entries d(e), rounded to T (apply_dinv's order) */
template <typename T, typename F>
__device__ __forceinline__ C3<T> cl_dinv(F d, C3<T> rv) {
    const double ra = rv.a, rb = rv.b, rc = rv.c;
    double z0 = 0.0, z1 = 0.0, z2 = 0.0;
    z0 = z0 + d(0) * ra; z0 = z0 + d(1) * rb; z0 = z0 + d(2) * rc;
    z1 = z1 + d(3) * ra; z1 = z1 + d(4) * rb; z1 = z1 + d(5) * rc;
    z2 = z2 + d(6) * ra; z2 = z2 + d(7) * rb; z2 = z2 + d(8) * rc;
    return { (T)z0, (T)z1, (T)z2 };
}

template <typename T>
__device__ __forceinline__ void cl_blk(const T *v, C3<T> p, T &q0, T &q1, T &q2) {
    q0 = q0 + v[0] * p.a;   q0 = q0 + v[32] * p.b;  q0 = q0 + v[64] * p.c;
    q1 = q1 + v[96] * p.a;  q1 = q1 + v[128] * p.b; q1 = q1 + v[160] * p.c;
    q2 = q2 + v[192] * p.a; q2 = q2 + v[224] * p.b; q2 = q2 + v[256] * p.c;
}

/* butterfly sum: lane 0's value is the shuffle-down tree's bit for bit (each step adds the
 * same two numbers, and addition is commutative), and every lane has it */
__device__ __forceinline__ double cl_warp_sum(double a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a = a + __shfl_xor_sync(0xffffffffu, a, o);
    return a;
}

__device__ __forceinline__ double cl_add(double a, double b) { return a + b; }
__device__ __forceinline__ double2 cl_add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double cl_xor(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ double2 cl_xor(double2 a, int o) { return make_double2(cl_xor(a.x, o), cl_xor(a.y, o)); }

/* the sum of the partials v[a] .. v[a + n - 1], n <= most <= 32 (most: the warp's largest n),
 * as the grid-wide solver's warp tree adds a CTA's warps (offsets 16, 8, 4, 2, 1; missing
 * warps are 0) */
template <int STRIDE>
__device__ __forceinline__ double cl_tree(const double *v, int a, int n, int most) {
    auto at = [&](int i) { return i < n ? v[STRIDE * (a + i)] : 0.0; };
    if (most <= 4) return (at(0) + at(2)) + (at(1) + at(3));
    double b[8];
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = most <= 8 ? at(i) : (at(i) + at(i + 16)) + (at(i + 8) + at(i + 24));
    return ((b[0] + b[4]) + (b[2] + b[6])) + ((b[1] + b[5]) + (b[3] + b[7]));
}
__device__ __forceinline__ double cl_tree(const double *v, int a, int n, int most) { return cl_tree<1>(v, a, n, most); }
__device__ __forceinline__ double2 cl_tree(const double2 *v, int a, int n, int most) {
    if (most <= 1) return n > 0 ? v[a] : make_double2(0.0, 0.0);
    return make_double2(cl_tree<2>(&v->x, a, n, most), cl_tree<2>(&v->y, a, n, most));
}

/* The sum of 16 values that every lane can read, on every lane, in the order of the butterfly
 * over 16 lanes: a lane adds the even or the odd ones in registers, and of double2 one
 * component (one or three shuffles instead of four or eight). */
__device__ __forceinline__ double cl_sum8(const double *v, int stride) {
    double b[8];
#pragma unroll
    for (int i = 0; i < 8; i++) b[i] = v[2 * i * stride];
    return ((b[0] + b[4]) + (b[2] + b[6])) + ((b[1] + b[5]) + (b[3] + b[7]));
}
__device__ __forceinline__ double cl_sum16(const double *v) {
    const double s = cl_sum8(v + (threadIdx.x & 1), 1);
    return s + cl_xor(s, 1);
}
__device__ __forceinline__ double2 cl_sum16(const double2 *v) {
    double s = cl_sum8(&v[threadIdx.x & 1].x + (threadIdx.x >> 1 & 1), 2);
    s = s + cl_xor(s, 1);
    return make_double2(__shfl_sync(0xffffffffu, s, 0), __shfl_sync(0xffffffffu, s, 2));
}

template <typename T> struct ClVec;
template <> struct ClVec<double> {
    static __device__ const double *val(const ClusterParams &P) { return P.val; }
    static __device__ const double *b(const ClusterParams &P) { return P.b4; }
    static __device__ double *x(const ClusterParams &P) { return P.x4; }
};
template <> struct ClVec<float> {
    static __device__ const float *val(const ClusterParams &P) { return P.val32; }
    static __device__ const float *b(const ClusterParams &P) { return P.bf4; }
    static __device__ float *x(const ClusterParams &P) { return P.xf4; }
};

/* U blocks of one row with values in shared memory: every load is issued before the first
 * sum (the warp's slots up to its slice's width exist, padded ones included; a shorter
 * row's lane leaves its sums alone) */
template <int U, typename T>
__device__ __forceinline__ void cl_blocks(const int *cb, const T *sv, const T *sp0, const T *sp1, const T *sp2, int left,
                                          T &q0, T &q1, T &q2) {
    int c[U];
    C3<T> p[U];
#pragma unroll
    for (int u = 0; u < U; u++) c[u] = cb[32 * u];
#pragma unroll
    for (int u = 0; u < U; u++) p[u] = C3<T>{ sp0[c[u]], sp1[c[u]], sp2[c[u]] };
#pragma unroll
    for (int u = 0; u < U; u++) {
        T n0 = q0, n1 = q1, n2 = q2;
        cl_blk(sv + 288 * u, p[u], n0, n1, n2);
        if (u < left) {
            q0 = n0;
            q1 = n1;
            q2 = n2;
        }
    }
}

__device__ __forceinline__ void cl_bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void cl_bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

/* ONE: the cluster is one CTA (its partials stay in its shared memory) */
template <typename T, int BS, int R, bool ONE, bool BATCH>
__global__ void __launch_bounds__(BS, 1) k_pcg_cluster(const ClusterParams P) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int MAXS = BS / 32 * R;                           /* slices of a CTA */
    constexpr int MAXP = MAXS <= 16 ? 16 : MAXS <= 32 ? 32 : 64; /* their partials, 0 beyond its slices */
    constexpr bool DREGS = R == 1;    /* the rows' D^-1 stay in registers, else L2 */
    constexpr int U = R == 1 ? 4 : 2; /* blocks whose loads are issued together */
    __shared__ __align__(8) uint64_t s_mb[3];            /* staging; p.q; r.z, r.r and halo z */
    __shared__ __align__(16) double s_part[MAXP];        /* the slices' p.q */
    __shared__ __align__(16) double2 s_part2[MAXP];      /* the slices' (r.z, r.r) */
    __shared__ __align__(16) double s_all[GSLAM_CLUSTER_CTAS];   /* the CTAs' p.q */
    __shared__ __align__(16) double2 s_all2[GSLAM_CLUSTER_CTAS]; /* the CTAs' (r.z, r.r) */
    __shared__ double s_bn, s_alpha, s_beta;
    /* 0 go on, else 1 + GSLAM_STOP_*: one word per reduction, because a warp may read the
     * first one while the second reduction is already being decided */
    __shared__ int s_flag_pq, s_flag;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
    const int C = ONE ? 1 : P.ctas, rank = ONE ? 0 : (int)cl_rank(), job = P.job0 + (int)blockIdx.x / C;
    const ClusterJob J = P.jobs[job];
    if (BATCH && P.skip != nullptr && __ldg(P.skip + J.graph)) return; /* the whole cluster */
    const int cta = J.cta0 + rank;
    const int s0 = __ldg(P.cta_slice + J.bound0 + rank), s1 = __ldg(P.cta_slice + J.bound0 + rank + 1), ns = s1 - s0;
    const int64_t slot0 = __ldg(P.slice_ptr + s0), slot1 = __ldg(P.slice_ptr + s1);
    const int n_halo = __ldg(P.n_halo + cta);
    const int n_loc = 32 * ns, row0 = 32 * s0;
    const ClusterSmem ml = cluster_smem_layout(sizeof(T), slot1 - slot0, ns, n_halo, J.halo_max, P.smem_budget);
    const int64_t nval = 9 * (slot1 - slot0), nsm = nval < ml.val_cap ? nval : ml.val_cap;
    unsigned char *zh = smem, *zh2 = smem + ml.zh2_off;
    int *scol = reinterpret_cast<int *>(smem + ml.col_off);
    const int np = n_loc + n_halo;
    T *sp0 = reinterpret_cast<T *>(smem + ml.p_off), *sp1 = sp0 + np, *sp2 = sp1 + np;
    T *sval = reinterpret_cast<T *>(smem + ml.val_off);
    const unsigned b_pq = cl_smem_u32(&s_mb[1]), b_rz = cl_smem_u32(&s_mb[2]);
    const unsigned a_zh = cl_smem_u32(zh), a_zh2 = cl_smem_u32(zh2);
    const unsigned bytes_pq = 8u * C, bytes_rz = 16u * C + (sizeof(T) == 8 ? 24u : 16u) * n_halo;
    auto arm = [&](unsigned bar, unsigned bytes) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    };

    /* ---- barriers, then this CTA's matrix share by TMA ---- */
    if (threadIdx.x == 0) {
        for (int i = 0; i < 3; i++) tma_mbar_init(&s_mb[i], 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (!ONE) {
            arm(b_pq, bytes_pq);
            arm(b_rz, bytes_rz);
        }
        s_flag = s_flag_pq = 0;
    }
    for (int i = threadIdx.x; i < MAXP; i += blockDim.x) {
        s_part[i] = 0.0;
        s_part2[i] = make_double2(0.0, 0.0);
    }
    if (threadIdx.x < GSLAM_CLUSTER_CTAS) {
        s_all[threadIdx.x] = 0.0; /* stay 0 beyond the cluster's CTAs */
        s_all2[threadIdx.x] = make_double2(0.0, 0.0);
    }
    /* every CTA's barriers are ready before anything is stored to it */
    if (ONE) __syncthreads();
    else cl_sync();
    const bool absent = rank == P.absent_cta; /* test hook: leaves without sending, the others time out */
    if (!absent && threadIdx.x == 0) {
        const unsigned vbytes = (unsigned)(sizeof(T) * nsm), cbytes = (unsigned)(4 * (slot1 - slot0));
        tma_mbar_expect_tx(&s_mb[0], vbytes + cbytes);
        /* one copy when every value fits, else one per slice (its kept positions) */
        if (nsm == nval) {
            if (vbytes) tma_bulk_g2s(sval, ClVec<T>::val(P) + 9 * slot0, vbytes, &s_mb[0]);
        } else {
            for (int t = s0; t < s1; t++) {
                const int n = __ldg(P.keep + t);
                if (n)
                    tma_bulk_g2s(sval + 288 * __ldg(P.pos + t), ClVec<T>::val(P) + 9 * __ldg(P.slice_ptr + t),
                                 (unsigned)(288 * sizeof(T)) * n, &s_mb[0]);
            }
        }
        if (cbytes) tma_bulk_g2s(scol, P.lcol + slot0, cbytes, &s_mb[0]);
        /* waited for by every thread below, after its first rows are read */
    }

    /* ---- this thread's rows ---- */
    int row[R], len[R], kept[R], spos[R], voff[R], e0[R], ecnt[R];
    bool mine[R];
    C3<T> x[R], r[R], z[R], p[R];
    double d[DREGS ? R : 1][9];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int s = s0 + warp + i * W;
        const bool own = s < s1;
        row[i] = 32 * s + lane;
        mine[i] = own && row[i] < P.n_rows;
        len[i] = mine[i] ? __ldg(P.row_len + row[i]) : 0;
        voff[i] = own ? (int)(__ldg(P.slice_ptr + s) - slot0) : 0;
        /* the slice's block positions with values in shared memory, and where; the last ones,
         * if they do not all fit, are read from L2 */
        kept[i] = own ? __ldg(P.keep + s) : 0;
        spos[i] = own ? 288 * __ldg(P.pos + s) : 0;
        const int er = J.exp0 + row[i] - 32 * J.slice0;
        e0[i] = mine[i] && !ONE ? __ldg(P.exp_ptr + er) : 0;
        ecnt[i] = mine[i] && !ONE ? __ldg(P.exp_ptr + er + 1) - e0[i] : 0;
        x[i] = r[i] = z[i] = p[i] = C3<T>{ 0, 0, 0 };
        if (DREGS && mine[i]) {
            const double *g = P.dinv + 288 * (size_t)s + lane;
#pragma unroll
            for (int e = 0; e < 9; e++) d[DREGS ? i : 0][e] = __ldg(g + 32 * e);
        }
    }
    auto dinv_row = [&](int i, C3<T> rv) {
        if (DREGS) return cl_dinv<T>([&](int e) { return d[DREGS ? i : 0][e]; }, rv);
        const double *g = P.dinv + 288 * (size_t)(row[i] >> 5) + lane;
        return cl_dinv<T>([&](int e) { return __ldg(g + 32 * e); }, rv);
    };
    /* z of an exported row to the CTAs that read it */
    auto send_z = [&]() {
        if constexpr (!ONE) {
#pragma unroll
            for (int i = 0; i < R; i++)
                for (int k = 0; k < ecnt[i]; k++) {
                    const unsigned code = __ldg(P.exp + e0[i] + k);
                    cl_send_z(a_zh, a_zh2, code >> 20, (int)(code & 0xfffffu), z[i], b_rz);
                }
        }
    };
    /* The sum over this CTA's slices, on every lane of the calling warp. ONE single graphs: in
     * the grid-wide solver's order, per CTA of its partition (lane c: its first slice and how
     * many), then over its CTAs; that butterfly runs over the next power of two of the CTAs
     * only: the steps left out would add zeros. */
    int p2 = 1, vt0 = 0, vtn = 0, vt_most = 0;
    if (ONE && !BATCH) {
        while (p2 < P.n_vcta) p2 *= 2;
        const int c = lane & (p2 - 1);
        if (c < P.n_vcta) {
            vt0 = __ldg(P.vcta_slice + c);
            vtn = __ldg(P.vcta_slice + c + 1) - vt0;
        }
        vt_most = __reduce_max_sync(0xffffffffu, vtn);
    }
    auto sum_slices = [&](const auto *v) {
        if constexpr (ONE && !BATCH) {
            auto s = cl_tree(v, vt0, vtn, vt_most);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                if (o < p2) s = cl_add(s, cl_xor(s, o));
            return s;
        } else if constexpr (MAXP == 16) {
            return cl_sum16(v);
        } else {
            auto s = v[lane];
            if (MAXP > 32) s = cl_add(s, v[(lane + 32) % MAXP]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s = cl_add(s, cl_xor(s, o));
            return s;
        }
    };

    bool ok = true;
    int k = 0, reason = GSLAM_STOP_MAXIT;
    /* The totals of p.q, and of (r.z, r.r), once every warp has left its slices' partials in
     * s_part or s_part2. ONE: on every lane of every warp, which then makes the scalars for
     * itself: one barrier per sum instead of three, 2.08 -> 1.57 us per iteration at 100 poses.
     * Else on the lanes of warp 0 only, because a wait that gives up has to be the whole CTA's:
     * one warp decides (and arms the barrier again, before it next stores to another CTA:
     * none can send the next sums earlier). `between` is the caller's work while the sums travel. */
    auto total_pq = [&]() {
        if (ONE) {
            __syncthreads();
            return sum_slices(s_part);
        }
        if (warp == 0) {
            cl_bar_sync(1, blockDim.x);
            const double s = sum_slices(s_part);
            if (lane < C) cl_st_async(cl_mapa(cl_smem_u32(&s_all[rank]), lane), s, cl_mapa(b_pq, lane));
        } else {
            cl_bar_arrive(1, blockDim.x);
        }
        if (warp != 0) return 0.0;
        ok = cl_wait(b_pq, k & 1, P.spin_limit);
        return cl_sum16(s_all);
    };
    auto total_rz = [&](auto between) {
        double2 t = make_double2(0.0, 0.0);
        if (ONE) {
            __syncthreads();
            t = sum_slices(s_part2);
            between();
            return t;
        }
        if (warp == 0) {
            cl_bar_sync(2, blockDim.x);
            t = sum_slices(s_part2);
            if (lane < C) cl_st_async2(cl_mapa(cl_smem_u32(&s_all2[rank]), lane), t.x, t.y, cl_mapa(b_rz, lane));
        } else {
            cl_bar_arrive(2, blockDim.x);
        }
        between();
        if (warp != 0) return t;
        ok = cl_wait(b_rz, k & 1, P.spin_limit);
        return cl_sum16(s_all2);
    };
    double rz_cur = 0.0, rr_cur = 0.0, limit = 0.0; /* ONE: in every thread; else in thread 0 */
    if (!absent) {
        /* ---- x = 0, r = b, z = D^-1 r; r.z and r.r ---- */
#pragma unroll
        for (int i = 0; i < R; i++) {
            double rz = 0.0, rr = 0.0;
            if (mine[i]) {
                r[i] = cl_ld_row(ClVec<T>::b(P), row[i]);
                z[i] = dinv_row(i, r[i]);
                const double r0 = r[i].a, r1 = r[i].b, r2 = r[i].c;
                rz = rz + r0 * (double)z[i].a; rz = rz + r1 * (double)z[i].b; rz = rz + r2 * (double)z[i].c;
                rr = rr + r0 * r0; rr = rr + r1 * r1; rr = rr + r2 * r2;
            }
            rz = cl_warp_sum(rz);
            rr = cl_warp_sum(rr);
            if (lane == 0 && warp + i * W < ns) s_part2[warp + i * W] = make_double2(rz, rr);
        }
        {
            const double2 t = total_rz(send_z);
            rz_cur = t.x;
            rr_cur = t.y;
            if (ONE || threadIdx.x == 0) limit = square_limit(P.tol_rel * sqrt(t.y));
            if (threadIdx.x == 0) {
                s_bn = sqrt(t.y);
                s_beta = 0.0;
                if (BATCH && t.y == 0.0) s_flag = 1 + GSLAM_STOP_TOL; /* zero right-hand side: x = 0 */
            }
            if (!ok) s_flag = 1 + GSLAM_STOP_TIMEOUT;
            else if (!ONE && threadIdx.x == 0) arm(b_rz, bytes_rz);
        }
        if (!tma_wait(&s_mb[0], 0, P.spin_limit)) {
            s_flag = 1 + GSLAM_STOP_TIMEOUT;
            tma_drain(&s_mb[0], 0);
        }
        __syncthreads();
        const int cap = BATCH && P.cap != nullptr ? min(P.max_iter, __ldg(P.cap + J.graph)) : P.max_iter;
        int flag = s_flag;
        T beta = (T)0;
        while (flag == 0) {
            if (k >= cap) break;
            /* ---- phase A: p = z + beta p, of own rows and (from its own copy) of the halo;
             *      q = A p; p.q ---- */
            if (!ONE) beta = (T)s_beta;
#pragma unroll
            for (int i = 0; i < R; i++)
                if (mine[i]) {
                    p[i] = k == 0 ? z[i] : C3<T>{ z[i].a + beta * p[i].a, z[i].b + beta * p[i].b, z[i].c + beta * p[i].c };
                    sp0[row[i] - row0] = p[i].a;
                    sp1[row[i] - row0] = p[i].b;
                    sp2[row[i] - row0] = p[i].c;
                }
            if (!ONE)
                for (int h = threadIdx.x; h < n_halo; h += blockDim.x) {
                    C3<T> hz = cl_halo_z<T>(zh, zh2, h);
                    T *h0 = sp0 + n_loc + h, *h1 = sp1 + n_loc + h, *h2 = sp2 + n_loc + h;
                    if (k > 0) hz = C3<T>{ hz.a + beta * *h0, hz.b + beta * *h1, hz.c + beta * *h2 };
                    *h0 = hz.a;
                    *h1 = hz.b;
                    *h2 = hz.c;
                }
            __syncthreads();
            C3<T> q[R];
#pragma unroll
            for (int i = 0; i < R; i++) {
                T q0 = 0, q1 = 0, q2 = 0;
                const int *cb = scol + voff[i] + lane;
                const T *sv = sval + spos[i] + lane;
                int j = 0;
                for (; j + U <= kept[i]; j += U)
                    cl_blocks<U>(cb + 32 * j, sv + 288 * j, sp0, sp1, sp2, len[i] - j, q0, q1, q2);
                if (U > 2 && kept[i] - j >= 2) {
                    cl_blocks<2>(cb + 32 * j, sv + 288 * j, sp0, sp1, sp2, len[i] - j, q0, q1, q2);
                    j += 2;
                }
                if (kept[i] - j >= 1) cl_blocks<1>(cb + 32 * j, sv + 288 * j, sp0, sp1, sp2, len[i] - j, q0, q1, q2);
                if (len[i] > kept[i]) {
                    /* the row's last blocks, from L2 */
                    const T *gv = ClVec<T>::val(P) + 9 * (slot0 + voff[i]) + lane;
                    for (j = kept[i]; j < len[i]; j++) {
                        T vb[9];
#pragma unroll
                        for (int e = 0; e < 9; e++) vb[e] = __ldg(gv + 288 * j + 32 * e);
                        const int c = cb[32 * j];
                        const C3<T> pc = { sp0[c], sp1[c], sp2[c] };
                        q0 = q0 + vb[0] * pc.a; q0 = q0 + vb[1] * pc.b; q0 = q0 + vb[2] * pc.c;
                        q1 = q1 + vb[3] * pc.a; q1 = q1 + vb[4] * pc.b; q1 = q1 + vb[5] * pc.c;
                        q2 = q2 + vb[6] * pc.a; q2 = q2 + vb[7] * pc.b; q2 = q2 + vb[8] * pc.c;
                    }
                }
                q[i] = C3<T>{ q0, q1, q2 };
                double pq = 0.0;
                if (mine[i]) {
                    pq = pq + (double)p[i].a * (double)q0; pq = pq + (double)p[i].b * (double)q1;
                    pq = pq + (double)p[i].c * (double)q2;
                }
                pq = cl_warp_sum(pq);
                if (lane == 0 && warp + i * W < ns) s_part[warp + i * W] = pq;
            }
            const double pq = total_pq();
            T alpha;
            if (ONE) {
                if (pq == 0.0) { flag = 1 + GSLAM_STOP_PQ_ZERO; break; }
                alpha = (T)(rz_cur / pq);
            } else {
                if (threadIdx.x == 0) {
                    if (!ok) s_flag_pq = 1 + GSLAM_STOP_TIMEOUT;
                    else if (pq == 0.0) s_flag_pq = 1 + GSLAM_STOP_PQ_ZERO;
                    s_alpha = rz_cur / pq;
                    if (ok) arm(b_pq, bytes_pq);
                }
                __syncthreads();
                flag = s_flag_pq;
                if (flag) break;
                alpha = (T)s_alpha;
            }
            /* ---- phase B: x += alpha p, r -= alpha q, z = D^-1 r; r.r and r.z ---- */
#pragma unroll
            for (int i = 0; i < R; i++) {
                double rr = 0.0, rz = 0.0;
                if (mine[i]) {
                    r[i] = C3<T>{ r[i].a - alpha * q[i].a, r[i].b - alpha * q[i].b, r[i].c - alpha * q[i].c };
                    z[i] = dinv_row(i, r[i]);
                    const double r0 = r[i].a, r1 = r[i].b, r2 = r[i].c;
                    rr = rr + r0 * r0; rr = rr + r1 * r1; rr = rr + r2 * r2;
                    rz = rz + r0 * (double)z[i].a; rz = rz + r1 * (double)z[i].b; rz = rz + r2 * (double)z[i].c;
                }
                double sums[2] = { rz, rr };
                const double sum = warp_sums<2>(sums);
                if ((lane & 15) == 0 && warp + i * W < ns) (&s_part2[warp + i * W].x)[lane >> 4] = sum;
            }
            k++;
            /* while the sums travel: the halo's z, and x */
            auto rest = [&]() {
                send_z();
#pragma unroll
                for (int i = 0; i < R; i++)
                    x[i] = C3<T>{ x[i].a + alpha * p[i].a, x[i].b + alpha * p[i].b, x[i].c + alpha * p[i].c };
            };
            const double2 t = total_rz(rest);
            if (ONE) {
                beta = (T)(t.x / rz_cur);
                rz_cur = t.x;
                rr_cur = t.y;
                if (t.y < limit) flag = 1 + GSLAM_STOP_TOL;
            } else {
                if (threadIdx.x == 0) {
                    if (!ok) s_flag = 1 + GSLAM_STOP_TIMEOUT;
                    else if (t.y < limit) s_flag = 1 + GSLAM_STOP_TOL;
                    s_beta = t.x / rz_cur;
                    rz_cur = t.x;
                    rr_cur = t.y;
                    if (ok) arm(b_rz, bytes_rz);
                }
                __syncthreads();
                flag = s_flag;
            }
        }
        if (flag) reason = flag - 1;
        if (reason == GSLAM_STOP_TIMEOUT && threadIdx.x == 0) res_mark_timeout(P.res);
#pragma unroll
        for (int i = 0; i < R; i++)
            if (mine[i]) cl_st_row(ClVec<T>::x(P), row[i], x[i]);
        if (rank == 0 && threadIdx.x == 0 && (BATCH || reason != GSLAM_STOP_TIMEOUT)) {
            PcgResult *res = BATCH ? P.gres + J.graph : P.res;
            res->iterations = k;
            res->refinements = 0;
            res->rnorm = sqrt(rr_cur);
            res->bnorm = s_bn;
            if (BATCH) res->reason = reason;
            else atomicCAS(&res->reason, 0, reason); /* another CTA's timeout stays */
        }
    }
    if (!ONE) {
        __syncthreads();
        cl_sync();
        if (absent || reason == GSLAM_STOP_TIMEOUT) {
            /* the others may have sent to this CTA up to their arrival above, in phases that it does
             * not wait for any more: 50 us for the last of that to land. A CTA that finished its
             * solve has received all that was sent to it. */
            const long long t0 = clock64();
            while (clock64() - t0 < 100000) {}
        }
    }
}

/* The kernel's shapes: up to 12, 16, 20 and 40 slices per CTA. One row per thread and 12 warps
 * have the registers for everything, 16 warps nearly (us per iteration in 384, 512, 640 threads:
 * 2.47, -, 2.59 at 5,120 poses; -, 2.99, 3.19 at 7,120); 20 warps (96 registers) hide more
 * latency than 10 warps of two rows each (64-graph batch: 11.1 ms of solve per round against
 * 12.9). */
template <typename T, bool ONE, bool BATCH>
static const void *fn_of(int shape) {
    switch (shape) {
    case 0: return (const void *)k_pcg_cluster<T, 384, 1, ONE, BATCH>;
    case 1: return (const void *)k_pcg_cluster<T, 512, 1, ONE, BATCH>;
    case 2: return (const void *)k_pcg_cluster<T, 640, 1, ONE, BATCH>;
    default: return (const void *)k_pcg_cluster<T, 640, 2, ONE, BATCH>;
    }
}

/* kinds of launches: 0 FP32 batches, 1 FP64 batches, 2 single graphs */
static const void *cluster_fn(int kind, int shape, bool one) {
    switch (kind) {
    case 0: return one ? fn_of<float, true, true>(shape) : fn_of<float, false, true>(shape);
    case 1: return one ? fn_of<double, true, true>(shape) : fn_of<double, false, true>(shape);
    default: return one ? fn_of<double, true, false>(shape) : fn_of<double, false, false>(shape);
    }
}

static void cluster_config(cudaLaunchConfig_t *cfg, cudaLaunchAttribute *at, int grid, int ctas, int threads,
                           size_t smem, cudaStream_t st) {
    *cfg = {};
    cfg->gridDim = dim3(grid);
    cfg->blockDim = dim3(threads);
    cfg->dynamicSmemBytes = smem;
    cfg->stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
}

cudaError_t launch_pcg_cluster(cudaStream_t st, const ClusterParams &p, int n_jobs, int threads, int shape,
                               size_t smem_bytes, bool fp32, bool batch) {
    if (n_jobs <= 0) return cudaSuccess;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    cluster_config(&cfg, at, n_jobs * p.ctas, p.ctas, threads, smem_bytes, st);
    ClusterParams copy = p;
    void *args[] = { &copy };
    const int kind = fp32 ? 0 : batch ? 1 : 2;
    return cudaLaunchKernelExC(&cfg, cluster_fn(kind, shape, p.ctas == 1), args);
}

int pcg_cluster_ctas(bool fp32, bool batch, int shape, int ctas, size_t smem_bytes) {
    const void *fn = cluster_fn(fp32 ? 0 : batch ? 1 : 2, shape, ctas == 1);
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    for (; ctas > 1; ctas /= 2) {
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at[1];
        cluster_config(&cfg, at, ctas, ctas, shape == 0 ? 384 : shape == 1 ? 512 : 640, smem_bytes, nullptr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) == cudaSuccess && n > 0) break;
        cudaGetLastError();
    }
    return ctas; /* one CTA needs no cluster */
}

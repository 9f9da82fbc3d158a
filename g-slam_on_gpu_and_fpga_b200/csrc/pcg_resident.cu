/*
 * pcg_resident.cu — the block-Jacobi PCG solver with the matrix resident in
 * shared memory (reference algorithm: src/cpu_pcg_fp64/MatrixOps.c:281-391).
 *
 * The solver's matrix does not change during a solve, and at the sizes this
 * back-end targets it fits in the GPU's aggregate shared memory (148 SMs x
 * 227 KB): N = 100,000 poses is ~211 KB of FP64 blocks per SM. So each CTA of a
 * cooperative launch (one per SM) copies its contiguous, slot-balanced share of
 * the sliced matrix into shared memory once, with TMA bulk copies
 * (cp.async.bulk, completion on an mbarrier), and every PCG iteration after that
 * reads values and column indices from shared memory. Of a share that does not fit
 * every slice leaves out its last block positions, which are read from L2: no
 * warp is then much slower than the others (whole slices in L2: 9.1 us per
 * iteration at N = 100,000 against 7.6 with one row per thread).
 *
 * A thread owns one or two block rows for the whole solve and keeps their x, r, z, p, q
 * and D^-1 in registers. Two rows per thread (12 warps) above 16 slices per CTA: with one
 * row, 768 threads have 80 registers each, which leaves D^-1 to L2 in every iteration
 * and spills; 6.9 us per iteration against 7.6 at N = 100,000 (1024 threads against 512
 * with two rows: 10.7 against 8.8 at 140,000).
 *
 * What crosses L2 in an iteration is z of the rows that other CTAs read (26 % at N =
 * 100,000), published with the iteration's number in the same 16-byte words, so that
 * its readers need no barrier and its writer no fence, and the CTAs' partial sums, sent
 * the same way (tag_reduce_*). p of a halo row is kept by its reader: the same z and
 * beta as its owner's give the same bits. Column indices are staged as CTA-local
 * indices: a CTA's own rows first, then its halo (the other CTAs' rows its blocks touch,
 * a list fixed at setup). Thread 0 alone advances the scalars (alpha, beta, the
 * stopping test) and hands them to the CTA through shared memory. Phases:
 *   A: p = z + beta p; q = A p; partial p.q                       -> grid reduction
 *   B: r -= alpha q; z = D^-1 r; partial r.r, r.z; x += alpha p   -> grid reduction
 * A published z needs one buffer: its owner overwrites it in phase B, after the sum of
 * p.q, which every reader enters after it has read the old one.
 *
 * Measured, us per iteration (before: a barrier counter with a release fence, p published
 * too, one row per thread): 3.15 (7.6) at N = 2,001, 3.5 (8.3) at 20,000, 4.25 (8.9) at
 * 50,000, 5.95 (12.7) at 100,000, 7.9 (16.6) at 140,000; the two all-reduces take about 2.5
 * of it. Sums and their order are unchanged, and so are the results' bits: each scalar row
 * of q adds its blocks in ascending original column order with separate multiply and add.
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gslam.h"
#include "kernels.cuh"
#include "pcg_common.cuh"
#include "tma_bulk.cuh"

/* U blocks of one row with values in shared memory, p at sp0 / sp1 / sp2: every load is issued
 * before the first sum (a warp's slots up to its slice's width exist, padded ones included; a
 * shorter row's lane leaves its sums alone) */
template <int U>
__device__ __forceinline__ void res_blocks(const int *cb, const double *sv, const double *sp0, const double *sp1,
                                           const double *sp2, int left, double &q0, double &q1, double &q2) {
    int c[U];
    V3 p[U];
#pragma unroll
    for (int u = 0; u < U; u++) c[u] = cb[32 * u];
#pragma unroll
    for (int u = 0; u < U; u++) p[u] = V3{ sp0[c[u]], sp1[c[u]], sp2[c[u]] };
#pragma unroll
    for (int u = 0; u < U; u++) {
        double n0 = q0, n1 = q1, n2 = q2;
        blk_acc_any(sv + 288 * u, p[u], n0, n1, n2);
        if (u < left) {
            q0 = n0;
            q1 = n1;
            q2 = n2;
        }
    }
}

/* R: slices per warp (warp w owns slices w and w + BS / 32); DREGS: the rows' D^-1 stay in
 * registers for the whole solve; U: blocks whose loads are issued together */
template <int BS, int R, bool DREGS, int U>
__global__ void __launch_bounds__(BS, 1) k_pcg64_res(PcgParams P) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int W = BS / 32;
    __shared__ double s_red[2][32];
    __shared__ double s_slot[2][TAG_LANES];
    __shared__ double s_bc[4];
    __shared__ int s_ok;
    /* scalars, advanced by thread 0 only: r.z, r.r, the limit of r.r; alpha and beta; stop
     * flags of the two reductions (1 + GSLAM_STOP_*) */
    __shared__ double s_rz, s_rr, s_limit, s_alpha, s_beta;
    __shared__ int s_flag_pq, s_flag;
    __shared__ __align__(8) uint64_t s_bar;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((int)blockIdx.x == P.absent_cta) return; /* test hook, see pcg.cu */

    const int s0 = __ldg(P.cta_slice + blockIdx.x), s1 = __ldg(P.cta_slice + blockIdx.x + 1);
    const int64_t slot0 = __ldg(P.slice_ptr + s0), slot1 = __ldg(P.slice_ptr + s1);
    const int64_t nval = 9 * (slot1 - slot0);
    const int n_loc = 32 * (s1 - s0), row0 = 32 * s0;
    const int h0 = __ldg(P.halo_ptr + blockIdx.x), n_halo = __ldg(P.halo_ptr + blockIdx.x + 1) - h0;
    /* this CTA's own layout (resident_smem_layout; the host checked that it fits): values as
     * far as they fit | local column indices | p of own + halo rows */
    const ResidentSmem ml = resident_smem_layout(slot1 - slot0, s1 - s0, n_halo, P.smem_budget);
    const int64_t nsm = nval < ml.val_cap ? nval : ml.val_cap; /* multiple of 288 */
    double *sval = reinterpret_cast<double *>(smem);
    int *scol = reinterpret_cast<int *>(smem + ml.col_off);
    double *sp0 = reinterpret_cast<double *>(smem + ml.p_off), *sp1 = sp0 + n_loc + n_halo, *sp2 = sp1 + n_loc + n_halo;

    /* ---- stage this CTA's matrix share ---- */
    if (threadIdx.x == 0) {
        tma_mbar_init(&s_bar, 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        s_ok = 1;
        s_flag = s_flag_pq = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        /* one copy when every value fits, else one per slice (its kept positions) */
        tma_mbar_expect_tx(&s_bar, (unsigned)(8 * nsm) + (unsigned)(4 * (slot1 - slot0)));
        if (slot1 > slot0) tma_bulk_g2s(scol, P.lcol + slot0, (unsigned)(4 * (slot1 - slot0)), &s_bar);
        if (nsm == nval) {
            if (nval) tma_bulk_g2s(sval, P.val + 9 * slot0, (unsigned)(8 * nval), &s_bar);
        } else {
            for (int t = s0; t < s1; t++) {
                const int keep = __ldg(P.res_keep + t);
                if (keep) tma_bulk_g2s(sval + 288 * __ldg(P.res_pos + t), P.val + 9 * __ldg(P.slice_ptr + t), 2304u * keep, &s_bar);
            }
        }
    }
    if (!tma_wait(&s_bar, 0, P.spin_limit)) {
        atomicExch(&P.gs->abort, 1);
        s_ok = 0;
        tma_drain(&s_bar, 0);
    }
    __syncthreads();
    if (!s_ok) {
        if (threadIdx.x == 0) res_mark_timeout(P.res);
        return;
    }

    /* ---- this thread's rows ---- */
    int row[R], len[R], kept[R], lslot[R], spos[R];
    bool mine[R], pub[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int s = s0 + warp + i * W;
        const bool own = s < s1;
        row[i] = 32 * s + lane;
        mine[i] = own && row[i] < P.n_rows;
        pub[i] = mine[i] && __ldg(P.row_export + row[i]); /* another CTA reads this row */
        len[i] = mine[i] ? __ldg(P.row_len + row[i]) : 0;
        lslot[i] = own ? (int)(__ldg(P.slice_ptr + s) - slot0) : 0; /* local slot of (j=0) */
        /* the slice's block positions with values in shared memory, and where; the last ones,
         * if they do not all fit, are read from L2 */
        kept[i] = own ? __ldg(P.res_keep + s) : 0;
        spos[i] = own ? 288 * __ldg(P.res_pos + s) : 0;
    }
    double d[DREGS ? R : 1][9];
    if (DREGS) {
#pragma unroll
        for (int i = 0; i < R; i++)
            if (mine[i]) {
                const double *g = P.dinv + 288 * (size_t)(row[i] >> 5) + lane;
#pragma unroll
                for (int e = 0; e < 9; e++) d[DREGS ? i : 0][e] = __ldg(g + 32 * e);
            }
    }
    auto precond = [&](int i, V3 v) {
        if (!DREGS) return apply_dinv(P.dinv, row[i], v);
        const double *e = d[DREGS ? i : 0];
        double z0 = 0.0, z1 = 0.0, z2 = 0.0;
        z0 = z0 + e[0] * v.a; z0 = z0 + e[1] * v.b; z0 = z0 + e[2] * v.c;
        z1 = z1 + e[3] * v.a; z1 = z1 + e[4] * v.b; z1 = z1 + e[5] * v.c;
        z2 = z2 + e[6] * v.a; z2 = z2 + e[7] * v.b; z2 = z2 + e[8] * v.c;
        return V3{ z0, z1, z2 };
    };

    /* the halo rows whose z this thread reads while the sums of r.r and r.z travel, the last
     * threads first (the first ten warps wait for the sums); further rows in phase A. Their p
     * is kept here too, beside the owner's, from the same z and beta, bit for bit. */
    const int hh = BS - 1 - (int)threadIdx.x;
    int hrow[R];
    V3 hz[R];
#pragma unroll
    for (int i = 0; i < R; i++) {
        hrow[i] = hh + i * BS < n_halo ? __ldg(P.halo_rows + h0 + hh + i * BS) : -1;
        hz[i] = V3{ 0.0, 0.0, 0.0 };
    }
    auto read_halo = [&](unsigned number) {
#pragma unroll
        for (int i = 0; i < R; i++)
            if (hrow[i] >= 0 && !tag_row_load(P.z4, hrow[i], number, P.gs, P.spin_limit, &hz[i])) s_ok = 0;
    };
    unsigned tag = 0; /* the reductions' numbers */

    V3 x[R], r[R], z[R], pn[R];
    {
        double acc2[2][R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            x[i] = r[i] = z[i] = pn[i] = V3{ 0.0, 0.0, 0.0 };
            acc2[0][i] = acc2[1][i] = 0.0;
            if (mine[i]) {
                r[i] = ldg3(P.b4, row[i]);
                z[i] = precond(i, r[i]);
                if (pub[i]) tag_row_store(P.z4, row[i], z[i], 1);
                double a = 0.0, b = 0.0;
                a = a + r[i].a * z[i].a; a = a + r[i].b * z[i].b; a = a + r[i].c * z[i].c;
                b = b + r[i].a * r[i].a; b = b + r[i].b * r[i].b; b = b + r[i].c * r[i].c;
                acc2[0][i] = a;
                acc2[1][i] = b;
            }
        }
        tag_reduce_send<2, R, BS>(acc2, P.tags, ++tag, s_red);
        tag_reduce_sum<2, BS>(P.tags, tag, P.gs, P.spin_limit, s_slot, s_bc, &s_ok);
        read_halo(1);
        if (threadIdx.x == 0) {
            s_rz = s_bc[0];
            s_rr = s_bc[1];
            s_limit = square_limit(P.tol_rel * sqrt(s_bc[1]));
            s_beta = 0.0;
            if (!s_ok) s_flag = 1 + GSLAM_STOP_TIMEOUT;
        }
        __syncthreads();
    }
    const double bnorm = sqrt(s_bc[1]);
    /* all threads read the same flag, as in the loop: s_ok may change at any time once a faster
     * warp polls halo rows, and a warp that left alone would be missed at the barriers */
    int k = 0, reason = GSLAM_STOP_MAXIT, flag = s_flag;

    while (!flag) {
        if (k >= P.max_iter) break;
        const double beta = s_beta;
        /* ---- phase A: p of own and halo rows into shared memory, then q = A p; p.q ---- */
#pragma unroll
        for (int i = 0; i < R; i++)
            if (mine[i]) {
                pn[i] = k == 0 ? z[i] : V3{ z[i].a + beta * pn[i].a, z[i].b + beta * pn[i].b, z[i].c + beta * pn[i].c };
                sp0[row[i] - row0] = pn[i].a;
                sp1[row[i] - row0] = pn[i].b;
                sp2[row[i] - row0] = pn[i].c;
            }
        auto halo_p = [&](int h, V3 v) {
            double *a = sp0 + n_loc + h, *b = sp1 + n_loc + h, *c = sp2 + n_loc + h;
            if (k > 0) v = V3{ v.a + beta * *a, v.b + beta * *b, v.c + beta * *c };
            *a = v.a;
            *b = v.b;
            *c = v.c;
        };
#pragma unroll
        for (int i = 0; i < R; i++)
            if (hrow[i] >= 0) halo_p(hh + i * BS, hz[i]);
        for (int h = hh + R * BS; h < n_halo; h += BS) {
            V3 v = { 0.0, 0.0, 0.0 };
            if (!tag_row_load(P.z4, __ldg(P.halo_rows + h0 + h), (unsigned)k + 1, P.gs, P.spin_limit, &v)) s_ok = 0;
            halo_p(h, v);
        }
        __syncthreads();
        V3 q[R];
        double pq[1][R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            double q0 = 0.0, q1 = 0.0, q2 = 0.0;
            const int *cb = scol + lslot[i] + lane;
            const double *sv = sval + spos[i] + lane;
            int j = 0;
            for (; j + U <= kept[i]; j += U) res_blocks<U>(cb + 32 * j, sv + 288 * j, sp0, sp1, sp2, len[i] - j, q0, q1, q2);
            if (U > 2 && kept[i] - j >= 2) {
                res_blocks<2>(cb + 32 * j, sv + 288 * j, sp0, sp1, sp2, len[i] - j, q0, q1, q2);
                j += 2;
            }
            if (U > 1 && kept[i] - j >= 1) res_blocks<1>(cb + 32 * j, sv + 288 * j, sp0, sp1, sp2, len[i] - j, q0, q1, q2);
            if (len[i] > kept[i]) {
                /* the row's last blocks, from L2 */
                auto ldp = [&](int c) { return V3{ sp0[c], sp1[c], sp2[c] }; };
                const double *gv = P.val + 9 * (slot0 + lslot[i]) + lane;
                for (j = kept[i]; j + 1 < len[i]; j += 2) {
                    const V3 p0 = ldp(cb[32 * j]), p1 = ldp(cb[32 * (j + 1)]);
                    blk_acc(gv + 288 * j, p0, q0, q1, q2);
                    blk_acc(gv + 288 * (j + 1), p1, q0, q1, q2);
                }
                if (j < len[i]) blk_acc(gv + 288 * j, ldp(cb[32 * j]), q0, q1, q2);
            }
            q[i] = V3{ q0, q1, q2 };
            pq[0][i] = 0.0;
            if (mine[i]) {
                pq[0][i] = pq[0][i] + pn[i].a * q0; pq[0][i] = pq[0][i] + pn[i].b * q1; pq[0][i] = pq[0][i] + pn[i].c * q2;
            }
        }
        tag_reduce_send<1, R, BS>(pq, P.tags, ++tag, s_red);
        tag_reduce_sum<1, BS>(P.tags, tag, P.gs, P.spin_limit, s_slot, s_bc, &s_ok);
        if (threadIdx.x == 0) {
            if (!s_ok) s_flag_pq = 1 + GSLAM_STOP_TIMEOUT;
            else if (s_bc[0] == 0.0) s_flag_pq = 1 + GSLAM_STOP_PQ_ZERO;
            s_alpha = s_rz / s_bc[0];
        }
        __syncthreads();
        flag = s_flag_pq;
        if (flag) break;
        const double alpha = s_alpha;
        /* ---- phase B: r -= alpha q; z = D^-1 r; r.r and r.z; x += alpha p ---- */
        double rs[2][R];
        k++;
#pragma unroll
        for (int i = 0; i < R; i++) {
            double rr = 0.0, rz = 0.0;
            if (mine[i]) {
                r[i] = V3{ r[i].a - alpha * q[i].a, r[i].b - alpha * q[i].b, r[i].c - alpha * q[i].c };
                z[i] = precond(i, r[i]);
                if (pub[i]) tag_row_store(P.z4, row[i], z[i], (unsigned)k + 1);
                rr = rr + r[i].a * r[i].a; rr = rr + r[i].b * r[i].b; rr = rr + r[i].c * r[i].c;
                rz = rz + r[i].a * z[i].a; rz = rz + r[i].b * z[i].b; rz = rz + r[i].c * z[i].c;
            }
            rs[0][i] = rr;
            rs[1][i] = rz;
        }
        tag_reduce_send<2, R, BS>(rs, P.tags, ++tag, s_red);
#pragma unroll
        for (int i = 0; i < R; i++)
            x[i] = V3{ x[i].a + alpha * pn[i].a, x[i].b + alpha * pn[i].b, x[i].c + alpha * pn[i].c };
        tag_reduce_sum<2, BS>(P.tags, tag, P.gs, P.spin_limit, s_slot, s_bc, &s_ok);
        if (threadIdx.x == 0) {
            const double rr = s_bc[0], rz_new = s_bc[1];
            s_rr = rr;
            if (!s_ok) s_flag = 1 + GSLAM_STOP_TIMEOUT;
            else if (rr < s_limit) s_flag = 1 + GSLAM_STOP_TOL;
            s_beta = rz_new / s_rz;
            s_rz = rz_new;
        }
        read_halo((unsigned)k + 1);
        __syncthreads();
        flag = s_flag;
    }
    if (flag) reason = flag - 1;
#pragma unroll
    for (int i = 0; i < R; i++)
        if (mine[i]) st3(P.x4, row[i], x[i]);
    if (reason == GSLAM_STOP_TIMEOUT && threadIdx.x == 0) {
        res_mark_timeout(P.res);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && reason != GSLAM_STOP_TIMEOUT) {
        res_finish(P.res, P.gs, k, reason, 0, sqrt(s_rr), bnorm);
    }
}

/* The kernel by the slices of the CTA that owns most: one or two per warp, and the largest
 * register share that leaves */
struct ResKernel {
    const void *fn;
    int block, max_slices;
};
static const ResKernel *res_kernels(int *n) {
    static const ResKernel k[] = {
        { (const void *)k_pcg64_res<384, 1, true, 4>, 384, 12 },
        { (const void *)k_pcg64_res<512, 1, true, 4>, 512, 16 },
        { (const void *)k_pcg64_res<384, 2, true, 2>, 384, 24 },
        { (const void *)k_pcg64_res<512, 2, false, 2>, 512, 32 },
    };
    *n = (int)(sizeof k / sizeof k[0]);
    return k;
}

cudaError_t launch_pcg_resident(cudaStream_t st, const PcgParams &p, int grid, int max_slices, size_t smem_bytes) {
    int n;
    const ResKernel *k = res_kernels(&n);
    for (int i = 0; i < n; i++)
        if (max_slices <= k[i].max_slices) {
            /* the attribute is per function and process: set once (pcg_resident_max_grid sets
             * it before any layout chooses this solver) */
            PcgParams copy = p;
            void *args[] = { &copy };
            return cudaLaunchCooperativeKernel(k[i].fn, dim3(grid), dim3(k[i].block), args, smem_bytes, st);
        }
    return cudaErrorInvalidValue;
}

int pcg_resident_max_grid(int device, size_t smem_bytes) {
    int n_sm = 0, best = 0, n;
    if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    const ResKernel *k = res_kernels(&n);
    for (int i = 0; i < n; i++) {
        int a = 0;
        if (cudaFuncSetAttribute(k[i].fn, cudaFuncAttributeMaxDynamicSharedMemorySize, GSLAM_GRID_SMEM_MAX) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k[i].fn, k[i].block, smem_bytes) != cudaSuccess)
            return 0;
        best = i == 0 ? a : std::min(best, a);
    }
    return best * n_sm;
}

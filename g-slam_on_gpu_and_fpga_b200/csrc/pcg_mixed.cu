/*
 * pcg_mixed.cu — mixed-precision solve of Omega dx = xi: FP32 inner block-Jacobi
 * PCG inside an FP64 iterative-refinement loop, one cooperative launch.
 *
 * Precisions (the reference solves everything in FP64: MatrixOps.c:281-391):
 *   FP64: the outer residual r = xi - Omega x (FP64 matrix), the solution x, every
 *         global dot product (accumulated in FP64), the 3x3 block inverses D^-1
 *         (stored and applied in FP64, the product rounded to FP32).
 *   FP32: the inner SpMV (FP32 copy of Omega, staged in shared memory), the inner
 *         vector updates and the inner correction d (x += d in FP64 after each
 *         inner solve).
 *
 * Inner iteration (Chronopoulos & Gear 1989, "s-step" CG with s = 1, in the
 * preconditioned form that also carries M^-1 of the recurrence vectors): with
 * s = A p, w = A z, u = M^-1 w and v = M^-1 s, alpha and beta come from ONE
 * fused reduction of (r.z, w.z, r.r) per iteration instead of the two of
 * standard PCG (M = the block diagonal, M^-1 = D^-1):
 *     s_{k-1} = w_{k-1} + beta s_{k-2};   v_{k-1} = u_{k-1} + beta v_{k-2}
 *     r_k = r_{k-1} - alpha s_{k-1};      z_k = z_{k-1} - alpha v_{k-1}
 *     p_{k-1} = z_{k-1} + beta p_{k-2};   d += alpha p_{k-1}
 *     w_k = A z_k;  u_k = D^-1 w_k;  gamma = r.z, delta = w.z, rho = r.r  -> reduction
 *     beta_k = gamma_k / gamma_{k-1};  alpha_k = gamma_k / (delta_k - beta_k gamma_k / alpha_{k-1})
 * (alpha, beta = those of the previous reduction). The SpMV needs z_k of rows
 * other CTAs own, which is only final after the reduction; instead of a second
 * grid barrier every row that another CTA reads publishes u_k before the
 * reduction, and its readers keep their own copies of its z and v and take the
 * owner's two FMAs per component, so the copies are bit-identical and no reader
 * needs the owner's D^-1. u is published with the iteration's number in the same
 * 16-byte words, and the sums travel the same way (tag_reduce_*): no fence, no
 * barrier counter. Two buffers of u alternate: an owner writes u_{k+2} after
 * reduction k + 1, which every reader enters after it has read u_k.
 *
 * Shared memory holds, per CTA: its matrix share (of a share that does not fit
 * every slice leaves out its last block positions, read from L2), CTA-local column
 * indices (own rows first, then the CTA's halo: the other CTAs' rows its blocks
 * touch, a list fixed at setup), z of its own and halo rows and the halo's v (of a halo
 * of thousands of rows, as far as it fits; the rest in global memory). Each
 * thread owns one or two rows and keeps r, z, s, v, w, u, p, d in registers, and
 * D^-1 where they suffice. Thread 0 alone advances the scalar recurrence while the
 * others fetch the halo's u. The SpMV reads values, columns and z from shared
 * memory only.
 *
 * Measured, us per iteration (before: a barrier counter with a release fence and z, u, v
 * of every row published), same bits. FP32: 2.7 (4.5) at N = 20,000, 2.7 (4.8) at 50,000,
 * 4.3 (5.9) at 100,000. FP64: 2.9 (6.2), 3.6 (7.6), 6.1 (11.8). Up to 50,000 the
 * all-reduce of three doubles (1.5 us) bounds it, at 100,000 the SpMV from shared memory
 * and, in FP64, D^-1 from L2.
 *
 * Outer step: x += d (FP64), grid barrier, r = xi - Omega x with the FP64 matrix,
 * ||r|| -> stop at tol * ||xi||, else restart the inner solve from r; a step that
 * does not halve ||r|| ends the solve with GSLAM_STOP_STAGNATION (the host then
 * solves in FP64).
 *
 * The same kernel with T = double is the FP64 one-reduction solver (GSLAM_PREC_FP64_CG):
 * one inner solve in FP64 to the outer tolerance and iteration cap, no refinement. It stops
 * on the recurrence residual, as the
 * reference's loop does (MatrixOps.c:345-347), and reports the true residual; its
 * iterates are the reference's PCG in exact arithmetic, with other rounding (20
 * Gauss-Newton rounds of a 100k-pose graph at 1e-6 / 500: 9.5e-10 from the reference
 * recurrence's poses, as close as a different summation order of that recurrence, 9.7e-10).
 */
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "gslam.h"
#include "kernels.cuh"
#include "pcg_common.cuh"
#include "tma_bulk.cuh"

/* a row's three components in the inner precision T; rows are padded to 4 elements
 * (16 B in FP32, 32 B in FP64) */
template <typename T> struct T3 { T a, b, c; };

__device__ __forceinline__ T3<float> ldcgt3(const float *v4, int row) {
    const float4 v = __ldcg(reinterpret_cast<const float4 *>(v4 + 4 * (size_t)row));
    return { v.x, v.y, v.z };
}
__device__ __forceinline__ T3<double> ldcgt3(const double *v4, int row) {
    const V3 v = ldcg3(v4, row);
    return { v.a, v.b, v.c };
}
__device__ __forceinline__ void stt3(float *v4, int row, T3<float> v) {
    *reinterpret_cast<float4 *>(v4 + 4 * (size_t)row) = make_float4(v.a, v.b, v.c, 0.f);
}
__device__ __forceinline__ void stt3(double *v4, int row, T3<double> v) { st3(v4, row, V3{ v.a, v.b, v.c }); }

/* a row published for the CTAs that read it, with the iteration's number: FP64 as
 * tag_row_store, FP32 as one 16-byte word */
__device__ __forceinline__ void put_row(double *v4, int row, T3<double> v, unsigned tag) {
    tag_row_store(v4, row, V3{ v.a, v.b, v.c }, tag);
}
__device__ __forceinline__ void put_row(float *v4, int row, T3<float> v, unsigned tag) {
    tag_store(reinterpret_cast<TagWord *>(v4 + 4 * (size_t)row),
              (unsigned long long)__float_as_uint(v.a) | (unsigned long long)__float_as_uint(v.b) << 32,
              (unsigned long long)__float_as_uint(v.c) | (unsigned long long)tag << 32);
}
__device__ __forceinline__ bool get_row(const double *v4, int row, unsigned tag, GridSync *gs, long long limit, T3<double> *v) {
    V3 t;
    if (!tag_row_load(v4, row, tag, gs, limit, &t)) return false;
    *v = T3<double>{ t.a, t.b, t.c };
    return true;
}
__device__ __forceinline__ bool get_row(const float *v4, int row, unsigned tag, GridSync *gs, long long limit, T3<float> *v) {
    const long long t0 = clock64();
    for (int n = 0;; n++) {
        const TagWord w = tag_load(reinterpret_cast<const TagWord *>(v4 + 4 * (size_t)row));
        if ((unsigned)(w.b >> 32) == tag) {
            *v = T3<float>{ __uint_as_float((unsigned)w.a), __uint_as_float((unsigned)(w.a >> 32)), __uint_as_float((unsigned)w.b) };
            return true;
        }
        if (tag_give_up(gs, n, t0, limit)) return false;
    }
}

/* z (and v) of own and halo rows in shared memory: FP32 one float4 per row, FP64 three arrays
 * (a gather of 8 bytes at stride 8 meets fewer bank conflicts than 16 + 8 bytes at stride 32) */
template <typename T> struct Rows;
template <> struct Rows<float> {
    float4 *p;
    __device__ Rows(unsigned char *at, int) : p(reinterpret_cast<float4 *>(at)) {}
    __device__ T3<float> get(int i) const { const float4 v = p[i]; return { v.x, v.y, v.z }; }
    __device__ void put(int i, T3<float> v) const { p[i] = make_float4(v.a, v.b, v.c, 0.f); }
};
template <> struct Rows<double> {
    double *a, *b, *c;
    __device__ Rows(unsigned char *at, int n) : a(reinterpret_cast<double *>(at)), b(a + n), c(b + n) {}
    __device__ T3<double> get(int i) const { return { a[i], b[i], c[i] }; }
    __device__ void put(int i, T3<double> v) const { a[i] = v.a; b[i] = v.b; c[i] = v.c; }
};

/* a * b + c in one rounding */
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }

/* y = D^-1 x in FP64 (the nine entries of D^-1), rounded to T. */
template <typename T>
__device__ __forceinline__ T3<T> dinv_apply_t(const double (&d)[9], T3<T> x) {
    const double x0 = x.a, x1 = x.b, x2 = x.c;
    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
    y0 = y0 + d[0] * x0; y0 = y0 + d[1] * x1; y0 = y0 + d[2] * x2;
    y1 = y1 + d[3] * x0; y1 = y1 + d[4] * x1; y1 = y1 + d[5] * x2;
    y2 = y2 + d[6] * x0; y2 = y2 + d[7] * x1; y2 = y2 + d[8] * x2;
    return T3<T>{ (T)y0, (T)y1, (T)y2 };
}

/* a * x + y, one FMA per component: every inner vector update */
template <typename T>
__device__ __forceinline__ T3<T> axpy_t(T a, T3<T> x, T3<T> y) {
    return T3<T>{ fma_t(a, x.a, y.a), fma_t(a, x.b, y.b), fma_t(a, x.c, y.c) };
}

/* v = u + beta v_old; z = z_old - alpha v: the step every copy of a row's z takes */
template <typename T>
__device__ __forceinline__ void step_zv(T3<T> z_old, T3<T> u, T3<T> v_old, T alpha, T beta, T3<T> &z_new,
                                        T3<T> &v_new) {
    v_new = axpy_t(beta, v_old, u);
    z_new = axpy_t(-alpha, v_new, z_old);
}

template <typename T>
__device__ __forceinline__ void blk_acc_t(const T *v, T3<T> p, T &q0, T &q1, T &q2) {
    q0 = fma_t(v[0], p.a, q0);   q0 = fma_t(v[32], p.b, q0);  q0 = fma_t(v[64], p.c, q0);
    q1 = fma_t(v[96], p.a, q1);  q1 = fma_t(v[128], p.b, q1); q1 = fma_t(v[160], p.c, q1);
    q2 = fma_t(v[192], p.a, q2); q2 = fma_t(v[224], p.b, q2); q2 = fma_t(v[256], p.c, q2);
}

/* U blocks of one row with values in shared memory: every load is issued before the first
 * sum (a shorter row's lane leaves its sums alone) */
template <int U, typename T>
__device__ __forceinline__ void mix_blocks(const int *cb, const T *sv, const Rows<T> &sz, int left, T &q0, T &q1, T &q2) {
    int c[U];
    T3<T> z[U];
#pragma unroll
    for (int u = 0; u < U; u++) c[u] = cb[32 * u];
#pragma unroll
    for (int u = 0; u < U; u++) z[u] = sz.get(c[u]);
#pragma unroll
    for (int u = 0; u < U; u++) {
        T n0 = q0, n1 = q1, n2 = q2;
        blk_acc_t(sv + 288 * u, z[u], n0, n1, n2);
        if (u < left) {
            q0 = n0;
            q1 = n1;
            q2 = n2;
        }
    }
}

/* the inner solve's buffers for T: the matrix copy, z at the start of an inner solve, and the
 * published u of both iteration parities */
template <typename T> struct Inner;
template <> struct Inner<float> {
    static __device__ const float *val(const PcgParams &P) { return P.val32; }
    static __device__ float *z0(const PcgParams &P) { return P.rf4; }
    static __device__ float *u(const PcgParams &P, unsigned par) { return par ? P.pfa4 : P.zf4; }
};
template <> struct Inner<double> {
    static __device__ const double *val(const PcgParams &P) { return P.val; }
    static __device__ double *z0(const PcgParams &P) { return P.r4; }
    static __device__ double *u(const PcgParams &P, unsigned par) { return par ? P.p4a : P.p4b; }
};

/* T = float: the mixed solver; T = double: the FP64 one-reduction solver (one inner solve).
 * R: slices per warp (warp w owns slices w and w + BS / 32); DREGS: the rows' D^-1 stay in
 * registers for the whole solve, else they are read from L2 in every iteration; U: blocks
 * whose loads are issued together; FAR: v of some halo rows is in global memory (kernels of their
 * own: the other layouts' lose up to 4 % to the registers it takes) */
template <int BS, int R, typename T, bool DREGS, int U, bool FAR>
__global__ void __launch_bounds__(BS, 1) k_pcg_mixed(PcgParams P) {
    constexpr bool F64 = sizeof(T) == 8;
    constexpr int W = BS / 32;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ double s_red[3][32];
    __shared__ double s_slot[3][TAG_LANES];
    __shared__ double s_bc[4];
    __shared__ int s_ok;
    __shared__ __align__(8) uint64_t s_bar;
    /* scalar recurrence, kept and advanced by thread 0 only (no registers in the
     * other threads): gamma_{k-1}, alpha_{k-1}, rho_0 of the inner solve, tol, ||xi|| */
    __shared__ double s_sc[5];
    __shared__ T s_ab[2];      /* alpha, beta for the next iteration */
    __shared__ int s_flag;     /* 0 continue, 1 inner solve done, 2 breakdown, 3 a wait gave up */
    __shared__ int s_conv;     /* the inner solve ended on its residual tolerance */
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int epoch = 0;
    unsigned seq = 0;          /* inner iterations so far: the number of their reduction and of u */
    if ((int)blockIdx.x == P.absent_cta) return; /* test hook, see pcg.cu */

    const int s0 = __ldg(P.cta_slice + blockIdx.x), s1 = __ldg(P.cta_slice + blockIdx.x + 1);
    const int row0 = 32 * s0, n_loc = 32 * (s1 - s0);
    const int64_t slot0 = __ldg(P.slice_ptr + s0), slot1 = __ldg(P.slice_ptr + s1);
    const int64_t nval = 9 * (slot1 - slot0);
    const int h0 = __ldg(P.halo_ptr + blockIdx.x), n_halo = __ldg(P.halo_ptr + blockIdx.x + 1) - h0;
    /* dynamic shared memory, laid out per CTA from its own sizes (mixed_smem_layout, the
     * host's feasibility check uses the same functions): T values as far as they fit |
     * local columns | z of own + halo rows | v of halo rows */
    const int n_shv = FAR ? (int)mixed_v_rows(sizeof(T), slot1 - slot0, s1 - s0, n_halo, R * BS, P.smem_budget) : n_halo;
    const MixedSmem ml = mixed_smem_layout(sizeof(T), slot1 - slot0, s1 - s0, n_halo, n_shv, P.smem_budget);
    const int64_t nsm = nval < ml.val_cap ? nval : ml.val_cap;
    T *sval = reinterpret_cast<T *>(smem);
    int *scol = reinterpret_cast<int *>(smem + ml.col_off);
    const Rows<T> sz(smem + ml.z_off, n_loc + n_halo), shv(smem + ml.v_off, n_shv);
    auto far_v = [&]() { return static_cast<T *>(P.halo_v); }; /* v of halo rows n_shv and up, at h0 + row */

    if (threadIdx.x == 0) {
        tma_mbar_init(&s_bar, 1);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        s_ok = 1;
    }
    __syncthreads();
    const int *keep = F64 ? P.cg_keep : P.mixed_keep, *pos = F64 ? P.cg_pos : P.mixed_pos;
    if (threadIdx.x == 0) {
        /* one copy when every value fits, else one per slice (its kept positions) */
        const unsigned vbytes = (unsigned)(sizeof(T) * nsm), cbytes = (unsigned)(4 * (slot1 - slot0));
        tma_mbar_expect_tx(&s_bar, vbytes + cbytes);
        if (cbytes) tma_bulk_g2s(scol, P.lcol + slot0, cbytes, &s_bar);
        if (nsm == nval) {
            if (vbytes) tma_bulk_g2s(sval, Inner<T>::val(P) + 9 * slot0, vbytes, &s_bar);
        } else {
            for (int t = s0; t < s1; t++) {
                const int n = __ldg(keep + t);
                if (n)
                    tma_bulk_g2s(sval + 288 * __ldg(pos + t), Inner<T>::val(P) + 9 * __ldg(P.slice_ptr + t),
                                 (unsigned)(288 * sizeof(T)) * n, &s_bar);
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
    double d9[DREGS ? R : 1][9];
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int s = s0 + warp + i * W;
        const bool own = s < s1;
        row[i] = 32 * s + lane;
        mine[i] = own && row[i] < P.n_rows;
        pub[i] = mine[i] && __ldg(P.row_export + row[i]); /* another CTA reads this row */
        len[i] = mine[i] ? __ldg(P.row_len + row[i]) : 0;
        lslot[i] = own ? (int)(__ldg(P.slice_ptr + s) - slot0) : 0;
        /* the slice's block positions with values in shared memory, and where; the last ones,
         * if they do not all fit, are read from L2 */
        kept[i] = own ? __ldg(keep + s) : 0;
        spos[i] = own ? 288 * __ldg(pos + s) : 0;
        if (DREGS && mine[i]) {
            const double *g = P.dinv + 288 * (size_t)(row[i] >> 5) + lane;
#pragma unroll
            for (int e = 0; e < 9; e++) d9[DREGS ? i : 0][e] = __ldg(g + 32 * e);
        }
    }
    auto precond = [&](int i, T3<T> v) {
        if (DREGS) return dinv_apply_t<T>(d9[DREGS ? i : 0], v);
        double d[9];
        const double *g = P.dinv + 288 * (size_t)(row[i] >> 5) + lane;
#pragma unroll
        for (int e = 0; e < 9; e++) d[e] = __ldg(g + 32 * e);
        return dinv_apply_t<T>(d, v);
    };
    /* the halo rows this thread advances, the last threads first (the first warps poll the
     * sums); further ones, when the halo has more rows than that, at the top of the iteration */
    const int hh = BS - 1 - (int)threadIdx.x;
    int hrow[R];
    T3<T> hu[R];
    const T3<T> zero = { (T)0, (T)0, (T)0 };
#pragma unroll
    for (int i = 0; i < R; i++) {
        hrow[i] = hh + i * BS < n_halo ? __ldg(P.halo_rows + h0 + hh + i * BS) : -1;
        hu[i] = zero;
    }

    /* ---- ||xi|| ---- */
    double bb[1] = { 0.0 };
    {
        double acc[1][R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            acc[0][i] = 0.0;
            if (mine[i]) {
                const V3 b = ldg3(P.b4, row[i]);
                acc[0][i] = acc[0][i] + b.a * b.a; acc[0][i] = acc[0][i] + b.b * b.b; acc[0][i] = acc[0][i] + b.c * b.c;
            }
        }
        if (!grid_allreduce_rows<1, R, BS>(acc, bb, P.partials, epoch, P.gs, P.spin_limit, s_red, s_bc, &s_ok)) {
            if (threadIdx.x == 0) res_mark_timeout(P.res);
            return;
        }
    }
    if (threadIdx.x == 0) {
        const double tol = P.tol_rel * sqrt(bb[0]);
        s_sc[3] = tol * tol;     /* compared with rho = r.r, so no square root per iteration */
        s_sc[4] = sqrt(bb[0]);
    }
    /* every thread reads s_sc[4] at the top of the loop: without this barrier a warp can take
     * an earlier kernel's value there for the norm, end its solve at once and leave the CTA's
     * other warps waiting for it at a barrier that counts warps */
    __syncthreads();

    /* FP64 solution (P.x4 holds it during an inner solve) and FP64 residual, = xi for x = 0;
     * the residual of the row is kept in P.q4 between refinement steps */
    double rnorm = sqrt(bb[0]);
    int total = 0, outer = 0, reason = GSLAM_STOP_MAXIT;
    bool timed_out = false;

    while (true) {
        if (rnorm < P.tol_rel * s_sc[4]) { reason = GSLAM_STOP_TOL; break; }
        if (total >= P.max_iter || outer >= P.max_refine) { reason = GSLAM_STOP_MAXIT; break; }
        outer++;
        /* ---- inner solve of A d = r64 in T; x += d in FP64 afterwards ---- */
        T3<T> r[R], z[R], w[R], u[R], sv[R], v[R], p[R], d[R];
#pragma unroll
        for (int i = 0; i < R; i++) {
            r[i] = z[i] = w[i] = u[i] = sv[i] = v[i] = p[i] = d[i] = zero;
            /* state "k = -1": z_{-1} = D^-1 r_0, and w, u, s, v, p of earlier steps 0, so with
             * alpha = beta = 0 the first step leaves r and z unchanged */
            if (mine[i]) {
                const V3 r64 = outer == 1 ? ldg3(P.b4, row[i]) : ld3(P.q4, row[i]);
                if (outer == 1) st3(P.x4, row[i], V3{ 0.0, 0.0, 0.0 });
                r[i] = T3<T>{ (T)r64.a, (T)r64.b, (T)r64.c };
                z[i] = precond(i, r[i]);
                if (pub[i]) stt3(Inner<T>::z0(P), row[i], z[i]);
            }
        }
        if (!grid_barrier(P.gs, (unsigned)(++epoch), P.spin_limit, &s_ok)) { timed_out = true; break; }
        for (int h = hh; h < n_halo; h += BS) {
            sz.put(n_loc + h, ldcgt3(Inner<T>::z0(P), __ldg(P.halo_rows + h0 + h)));
            if (!FAR || h < n_shv) shv.put(h, zero);
            else stt3(far_v(), h0 + h, zero);
        }
#pragma unroll
        for (int i = 0; i < R; i++) hu[i] = zero;
        T alpha = (T)0, beta = (T)0;
        int k = 0;
        while (true) {
            /* z_k of the halo rows, from the owners' u_{k-1} and this CTA's copies of v and z:
             * the owners' own step, bit for bit */
            auto halo_step = [&](int h, T3<T> uh) {
                T3<T> zn, vn;
                step_zv(sz.get(n_loc + h), uh, shv.get(h), alpha, beta, zn, vn);
                sz.put(n_loc + h, zn);
                shv.put(h, vn);
            };
#pragma unroll
            for (int i = 0; i < R; i++)
                if (hrow[i] >= 0) halo_step(hh + i * BS, hu[i]);
            for (int h = hh + R * BS; h < n_halo; h += BS) {
                T3<T> uh = zero;
                if (k > 0 && !get_row(Inner<T>::u(P, seq & 1), __ldg(P.halo_rows + h0 + h), seq, P.gs, P.spin_limit, &uh)) s_ok = 0;
                if (!FAR || h < n_shv) {
                    halo_step(h, uh);
                } else {
                    T3<T> zn, vn;
                    step_zv(sz.get(n_loc + h), uh, ldcgt3(far_v(), h0 + h), alpha, beta, zn, vn);
                    sz.put(n_loc + h, zn);
                    stt3(far_v(), h0 + h, vn);
                }
            }
            /* own rows: s_{k-1}, r_k, p_{k-1}, d, then v_{k-1}, z_k */
#pragma unroll
            for (int i = 0; i < R; i++) {
                sv[i] = axpy_t(beta, sv[i], w[i]);
                r[i] = axpy_t(-alpha, sv[i], r[i]);
                p[i] = axpy_t(beta, p[i], z[i]);
                if (k > 0) d[i] = axpy_t(alpha, p[i], d[i]);
                step_zv(z[i], u[i], v[i], alpha, beta, z[i], v[i]);
                if (mine[i]) sz.put(row[i] - row0, z[i]);
            }
            __syncthreads();
            seq++;
            /* w_k = A z_k from shared memory, u_k = D^-1 w_k */
            double part[3][R];
#pragma unroll
            for (int i = 0; i < R; i++) {
                T q0 = (T)0, q1 = (T)0, q2 = (T)0;
                const int *cb = scol + lslot[i] + lane;
                const T *sv0 = sval + spos[i] + lane;
                int j = 0;
                for (; j + U <= kept[i]; j += U) mix_blocks<U, T>(cb + 32 * j, sv0 + 288 * j, sz, len[i] - j, q0, q1, q2);
                if (U > 2 && kept[i] - j >= 2) {
                    mix_blocks<2, T>(cb + 32 * j, sv0 + 288 * j, sz, len[i] - j, q0, q1, q2);
                    j += 2;
                }
                if (U > 1 && kept[i] - j >= 1) mix_blocks<1, T>(cb + 32 * j, sv0 + 288 * j, sz, len[i] - j, q0, q1, q2);
                if (len[i] > kept[i]) {
                    /* the row's last blocks, from L2 */
                    const T *gv = Inner<T>::val(P) + 9 * (slot0 + lslot[i]) + lane;
                    for (j = kept[i]; j < len[i]; j++) {
                        T vb[9];
#pragma unroll
                        for (int e = 0; e < 9; e++) vb[e] = __ldg(gv + 288 * j + 32 * e);
                        const T3<T> zc = sz.get(cb[32 * j]);
                        q0 = fma_t(vb[0], zc.a, q0); q0 = fma_t(vb[1], zc.b, q0); q0 = fma_t(vb[2], zc.c, q0);
                        q1 = fma_t(vb[3], zc.a, q1); q1 = fma_t(vb[4], zc.b, q1); q1 = fma_t(vb[5], zc.c, q1);
                        q2 = fma_t(vb[6], zc.a, q2); q2 = fma_t(vb[7], zc.b, q2); q2 = fma_t(vb[8], zc.c, q2);
                    }
                }
                part[0][i] = part[1][i] = part[2][i] = 0.0;
                if (mine[i]) {
                    w[i] = T3<T>{ q0, q1, q2 };
                    u[i] = precond(i, w[i]);
                    if (pub[i]) put_row(Inner<T>::u(P, seq & 1), row[i], u[i], seq);
                    const double r0 = r[i].a, r1 = r[i].b, r2 = r[i].c, z0 = z[i].a, z1 = z[i].b, z2 = z[i].c;
                    part[0][i] = r0 * z0 + r1 * z1 + r2 * z2;                                           /* gamma */
                    part[1][i] = (double)w[i].a * z0 + (double)w[i].b * z1 + (double)w[i].c * z2;       /* delta */
                    part[2][i] = r0 * r0 + r1 * r1 + r2 * r2;                                           /* rho */
                }
            }
            tag_reduce_send<3, R, BS>(part, P.tags, seq, s_red);
            tag_reduce_sum<3, BS>(P.tags, seq, P.gs, P.spin_limit, s_slot, s_bc, &s_ok);
            total++;
            k++;
            if (threadIdx.x == 0) {
                /* alpha_k = gamma / (delta - beta_k gamma / alpha_{k-1}) = gamma g / (delta g - gamma^2)
                 * with g = gamma_{k-1} alpha_{k-1}: one FP64 division on the critical path (beta's
                 * runs beside it); both rounded to T for the vector updates */
                const double gamma = s_bc[0], delta = s_bc[1], rho = s_bc[2];
                if (k == 1) s_sc[2] = rho;
                double a, bt;
                if (k == 1) { bt = 0.0; a = gamma / delta; }
                else {
                    const double g = s_sc[0] * s_sc[1];
                    bt = gamma / s_sc[0];
                    a = (gamma * g) / (delta * g - gamma * gamma);
                }
                int flag = 0, conv = 0;
                if (!s_ok) flag = 3;
                else if (!(delta != 0.0) || !(a == a) || isinf(a)) flag = 2;
                else if (rho <= P.inner_tol * P.inner_tol * s_sc[2] || rho < s_sc[3])
                    flag = conv = 1;
                else if (k >= P.inner_max_iter || total >= P.max_iter)
                    flag = 1;
                s_conv = conv;
                s_sc[0] = gamma;
                s_sc[1] = a;
                s_ab[0] = (T)a;
                s_ab[1] = (T)bt;
                s_flag = flag;
            }
            /* the halo's u_k, while the sums are made */
#pragma unroll
            for (int i = 0; i < R; i++)
                if (hrow[i] >= 0 && !get_row(Inner<T>::u(P, seq & 1), hrow[i], seq, P.gs, P.spin_limit, &hu[i])) s_ok = 0;
            __syncthreads();
            const int flag = s_flag;
            if (flag == 3) { timed_out = true; break; }
            if (flag == 2) { reason = GSLAM_STOP_PQ_ZERO; break; }
            alpha = s_ab[0];
            beta = s_ab[1];
            if (flag == 1) {
                /* the last update: d += alpha_k p_k, p_k = z_k + beta_k p_{k-1}. The FP64
                 * solve that met its tolerance ends without it, at the solution whose
                 * residual met the test (the reference's loop stops there); its step count is
                 * one less than its reductions. */
                if (F64 && s_conv) {
                    total--;
                } else {
#pragma unroll
                    for (int i = 0; i < R; i++) {
                        p[i] = axpy_t(beta, p[i], z[i]);
                        d[i] = axpy_t(alpha, p[i], d[i]);
                    }
                }
                break;
            }
        }
        if (timed_out) break;
        /* ---- x += d in FP64, then the outer FP64 residual r64 = xi - A x ---- */
#pragma unroll
        for (int i = 0; i < R; i++)
            if (mine[i]) {
                const V3 x = ld3(P.x4, row[i]);
                st3(P.x4, row[i], V3{ x.a + (double)d[i].a, x.b + (double)d[i].b, x.c + (double)d[i].c });
            }
        if (!grid_barrier(P.gs, (unsigned)(++epoch), P.spin_limit, &s_ok)) { timed_out = true; break; }
        double acc[1][R], rr[1] = { 0.0 };
#pragma unroll
        for (int i = 0; i < R; i++) {
            acc[0][i] = 0.0;
            if (mine[i]) {
                const int64_t sb = slot0 + lslot[i];
                const V3 ax = spmv_row(P.val + 9 * sb + lane, P.col + sb + lane, len[i], P.x4, P.x4, 0.0, true);
                const V3 b = ldg3(P.b4, row[i]);
                const V3 r64 = V3{ b.a - ax.a, b.b - ax.b, b.c - ax.c };
                if (!F64) st3(P.q4, row[i], r64);
                acc[0][i] = acc[0][i] + r64.a * r64.a; acc[0][i] = acc[0][i] + r64.b * r64.b; acc[0][i] = acc[0][i] + r64.c * r64.c;
            }
        }
        if (!grid_allreduce_rows<1, R, BS>(acc, rr, P.partials, epoch, P.gs, P.spin_limit, s_red, s_bc, &s_ok)) {
            timed_out = true;
            break;
        }
        const double rnorm_prev = rnorm;
        rnorm = sqrt(rr[0]);
        if (reason == GSLAM_STOP_PQ_ZERO) break;
        if (F64) {
            /* one FP64 solve: TOL if its recurrence residual met the tolerance, else the
             * iteration cap */
            reason = s_conv ? GSLAM_STOP_TOL : GSLAM_STOP_MAXIT;
            break;
        }
        /* iterative refinement must shrink the true residual; when a step gains less than a
         * factor 2 the FP32 inner solve cannot resolve this system (cond x eps32 >> 1) */
        if (rnorm >= P.tol_rel * s_sc[4] && total < P.max_iter && outer < P.max_refine &&
            rnorm > 0.5 * rnorm_prev) {
            reason = GSLAM_STOP_STAGNATION;
            break;
        }
    }
    /* P.x4 already holds x: stored at the start of the first refinement step and after each; a
     * solve that needs none stores its zeros here */
    if (outer == 0)
#pragma unroll
        for (int i = 0; i < R; i++)
            if (mine[i]) st3(P.x4, row[i], V3{ 0.0, 0.0, 0.0 });
    if (timed_out && threadIdx.x == 0) {
        res_mark_timeout(P.res);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && !timed_out) {
        res_finish(P.res, P.gs, total, reason, outer, rnorm, s_sc[4]);
    }
}

/* The kernel by precision and by the slices of the CTA that owns most: one or two per warp, as
 * leaves registers for the rows' state. Us per iteration: FP32 at 56,000 poses (18 slices)
 * 3.27 with one row per thread, 3.76 with two; at 70,000 (22) 4.40 (768 threads, spills) and
 * 4.33; at 140,000 (32) 5.75 (1024 threads) and 5.24. FP64 at 56,000 5.26 (768 threads) and
 * 4.52, at 100,000 6.88 and 6.31; D^-1 loaded ahead of the product instead of after it
 * spills: 8.1. */
struct MixKernel {
    const void *fn, *far; /* far: some halo rows' v in global memory */
    int block, max_slices;
};
template <int BS, int R, typename T, bool DREGS, int U>
static MixKernel mix_kernel() {
    return { (const void *)k_pcg_mixed<BS, R, T, DREGS, U, false>, (const void *)k_pcg_mixed<BS, R, T, DREGS, U, true>, BS,
             R * BS / 32 };
}
static const MixKernel *mix_kernels(bool fp64, int *n) {
    static const MixKernel f[] = {
        mix_kernel<384, 1, float, true, 4>(), mix_kernel<512, 1, float, true, 4>(), mix_kernel<640, 1, float, true, 4>(),
        mix_kernel<384, 2, float, true, 4>(), mix_kernel<512, 2, float, false, 2>(),
    };
    static const MixKernel d[] = {
        mix_kernel<384, 1, double, true, 4>(), mix_kernel<512, 1, double, true, 2>(), mix_kernel<384, 2, double, false, 4>(),
        mix_kernel<512, 2, double, false, 1>(),
    };
    *n = (int)(fp64 ? sizeof d / sizeof d[0] : sizeof f / sizeof f[0]);
    return fp64 ? d : f;
}

int pcg_mixed_rows(bool fp64, int max_slices) {
    int n;
    const MixKernel *k = mix_kernels(fp64, &n);
    for (int i = 0; i < n; i++)
        if (max_slices <= k[i].max_slices) return 32 * k[i].max_slices;
    return 0;
}

cudaError_t launch_pcg_mixed(cudaStream_t st, const PcgParams &p, int grid, int max_slices, size_t smem_bytes, bool fp64) {
    int n;
    const MixKernel *k = mix_kernels(fp64, &n);
    for (int i = 0; i < n; i++)
        if (max_slices <= k[i].max_slices) {
            PcgParams copy = p;
            void *args[] = { &copy };
            return cudaLaunchCooperativeKernel(p.halo_v ? k[i].far : k[i].fn, dim3(grid), dim3(k[i].block), args, smem_bytes, st);
        }
    return cudaErrorInvalidValue;
}

int pcg_mixed_max_grid(int device, size_t smem_bytes) {
    int n_sm = 0, best = 0, n;
    if (cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    for (int f = 0; f < 2; f++) {
        const MixKernel *k = mix_kernels(f != 0, &n);
        for (int i = 0; i < n; i++)
            for (const void *fn : { k[i].fn, k[i].far }) {
                int a = 0;
                if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, GSLAM_GRID_SMEM_MAX) != cudaSuccess ||
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, fn, k[i].block, smem_bytes) != cudaSuccess)
                    return 0;
                best = f == 0 && i == 0 && fn == k[i].fn ? a : std::min(best, a);
            }
    }
    return best * n_sm;
}

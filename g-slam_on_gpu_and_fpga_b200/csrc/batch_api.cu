/*
 * batch_api.cu — the batch entry points of the handle API (include/gslam.h):
 * gslam_create_se2_batch, gslam_batch_round, gslam_batch_layout, and the batched
 * solves behind gslam_solve / gslam_round on a batch handle.
 *
 * No counterpart in the reference, which solves one graph per process and sweeps
 * lambda with a shell loop (README.md:137-160). A batch is one block-diagonal graph:
 * every graph's poses padded to whole 32-row slices, its own lambda and anchor, its own
 * PCG scalars: in a thread-block cluster of its own (pcg_cluster.cu), or all of them in one
 * persistent launch of batch.cu's solver.
 */
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "cluster_plan.h"
#include "gslam.h"
#include "gslam_api_internal.h"
#include "gslam_internal.h"
#include "kernels.cuh"
#include "pcg_common.cuh"

/* batches of SE(2) graphs (one block-diagonal graph, batch.cu's solver)     */
/* ------------------------------------------------------------------------ */

static int batch_clusters_build(gslam_graph *g, bool fp32);

/* CTA shapes of 12, 20 and 40 slices: the 16-slice one would only split the launches further
 * (solve of the 64 graphs below, ms: 8.9 without it, 9.6 with it; 9.1 without the 12-slice one) */
#define GSLAM_BATCH_SHAPES 13u

static int batch_partition(gslam_graph *g) {
    BatchState &B = *g->batch;
    const gslam_structure &S = g->S;
    DevMem &m = g->mem;
    int n_sm = 0;
    CK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, g->device));
    B.block = g->o.threads_per_cta ? g->o.threads_per_cta : 512;
    const int cps = g->o.ctas_per_sm ? g->o.ctas_per_sm : 2; /* two 64-register CTAs per SM by default */
    const int warps = B.block / 32;
    /* slices per CTA: room to balance by slot count, at least one per warp */
    int grid_guess = cps * n_sm;
    B.max_slices = std::max(warps, 2 * ((S.n_slices + grid_guess - 1) / grid_guess));
    B.smem_bytes = 2 * sizeof(double) * (size_t)B.max_slices;
    const int maxg = pcg_batch_max_grid(B.block, B.smem_bytes, g->device);
    if (maxg <= 0) {
        gslam_set_last_error("batched solver cannot be made co-resident at this block size");
        return GSLAM_ERR_NO_DEVICE;
    }
    const int grid = std::max(1, std::min(maxg, grid_guess));
    B.max_slices = std::max(B.max_slices, (S.n_slices + grid - 1) / grid);
    B.smem_bytes = 2 * sizeof(double) * (size_t)B.max_slices;
    /* contiguous ranges of at most max_slices slices minimising the largest slot count */
    const int cap = B.max_slices;
    auto fill = [&](int64_t bound, std::vector<int> *out) {
        int used = 1, nsl = 0;
        int64_t cur = 0;
        if (out) (*out)[0] = 0;
        for (int sl = 0; sl < S.n_slices; sl++) {
            const int64_t w = S.slice_ptr[sl + 1] - S.slice_ptr[sl];
            if (nsl > 0 && (cur + w > bound || nsl == cap)) {
                if (out && used <= grid) (*out)[used] = sl;
                used++;
                cur = 0;
                nsl = 0;
            }
            cur += w;
            nsl++;
        }
        if (out)
            for (int i = std::min(used, grid); i <= grid; i++) (*out)[i] = S.n_slices;
        return used;
    };
    int64_t lo = 0, hi = S.n_slots;
    for (int sl = 0; sl < S.n_slices; sl++) lo = std::max(lo, S.slice_ptr[sl + 1] - S.slice_ptr[sl]);
    while (lo < hi) {
        const int64_t mid = lo + (hi - lo) / 2;
        if (fill(mid, nullptr) <= grid) hi = mid;
        else lo = mid + 1;
    }
    std::vector<int> cs(grid + 1);
    fill(lo, &cs);
    if (cs[grid] != S.n_slices) { gslam_set_last_error("batch partition failed"); return GSLAM_ERR_TOO_LARGE; }
    B.grid = grid;
    /* graph of each slice; graphs of each CTA; CTAs of each graph */
    const int G = B.n_graphs;
    std::vector<int> slice_graph(S.n_slices, 0);
    for (int q = 0; q < G; q++)
        for (int sl = B.pose_off[q] / 32; sl < B.pose_off[q + 1] / 32; sl++) slice_graph[sl] = q;
    std::vector<int> g0(grid, 0), g1(grid, -1), gc0(G, -1), gnc(G, 0), poff(G, 0);
    for (int c = 0; c < grid; c++) {
        if (cs[c + 1] <= cs[c]) continue;
        g0[c] = slice_graph[cs[c]];
        g1[c] = slice_graph[cs[c + 1] - 1];
        if (g1[c] - g0[c] + 1 > pcg_batch_lg_max()) {
            gslam_set_last_error("too many small graphs per CTA for the batched solver");
            return GSLAM_ERR_TOO_LARGE;
        }
        for (int q = g0[c]; q <= g1[c]; q++) {
            if (gc0[q] < 0) gc0[q] = c;
            gnc[q]++;
        }
    }
    int total = 0;
    for (int q = 0; q < G; q++) { poff[q] = total; total += gnc[q]; }
    B.total_parts = total;
    CK(dupload(m, g->st, &B.d_cta_slice, cs));
    CK(dupload(m, g->st, &B.d_slice_graph, slice_graph));
    CK(dupload(m, g->st, &B.d_cta_g0, g0));
    CK(dupload(m, g->st, &B.d_cta_g1, g1));
    CK(dupload(m, g->st, &B.d_graph_cta0, gc0));
    CK(dupload(m, g->st, &B.d_graph_ncta, gnc));
    CK(dupload(m, g->st, &B.d_part_off, poff));
    CK(dalloc(m, &B.d_partials, 4 * (size_t)std::max(total, 1)));
    return GSLAM_OK;
}

int gslam_create_se2_batch(const gslam_se2_graph *graphs, uint32_t n_graphs, const gslam_opts *opts,
                           gslam_graph **out) {
    if (!graphs || !out || n_graphs == 0) BAD("null argument or empty batch");
    *out = nullptr;
    int64_t total = 0, n_edges = 0;
    for (uint32_t q = 0; q < n_graphs; q++) {
        const gslam_se2_graph &in = graphs[q];
        if (in.n_poses == 0 || !in.poses) BAD("a graph of the batch has no poses");
        if (in.n_edges && (!in.edge_i || !in.edge_j || !in.meas || !in.log_w)) BAD("missing edge arrays");
        for (uint32_t e = 0; e < in.n_edges; e++)
            if (in.edge_i[e] >= in.n_poses || in.edge_j[e] >= in.n_poses) BAD("edge pose out of range");
        if (!(in.lambda > 0.0)) BAD("lambda must be positive");
        total += ((int64_t)in.n_poses + 31) / 32 * 32;
        n_edges += in.n_edges;
    }
    if (total > 0x3fffffff || n_edges > 0x7fffffff) { gslam_set_last_error("batch too large"); return GSLAM_ERR_TOO_LARGE; }
    gslam_graph *g = new gslam_graph();
    int rc = common_setup(g, opts);
    if (rc != GSLAM_OK) { gslam_destroy(g); return rc; }
    auto fail = [&](int code) { gslam_destroy(g); return code; };
    g->batch = new BatchState();
    BatchState &B = *g->batch;
    B.n_graphs = (int)n_graphs;
    g->factors = GSLAM_FACTORS_SE2;
    g->n_poses = (int)total;
    g->lambda = 1.0;        /* each graph's lambda is folded into its information weights */
    g->anchor = 0.0;
    g->n_obs_edges = 0;
    g->n_edges = n_edges;
    B.pose_off.assign(n_graphs + 1, 0);
    B.n_real.assign(n_graphs, 0);
    std::vector<unsigned> t1, t2;
    std::vector<double> meas, info, poses(3 * (size_t)total, 0.0), anchor_vals;
    std::vector<int> diag_rows, segments, anchor_rows;
    t1.reserve(n_edges); t2.reserve(n_edges);
    meas.reserve(3 * n_edges); info.reserve(3 * n_edges);
    for (uint32_t q = 0; q < n_graphs; q++) {
        const gslam_se2_graph &in = graphs[q];
        const int off = B.pose_off[q];
        const int padded = (int)((in.n_poses + 31) / 32 * 32);
        B.pose_off[q + 1] = off + padded;
        B.n_real[q] = (int)in.n_poses;
        B.max_chunks = std::max(B.max_chunks, batch_max_chunks(padded));
        segments.push_back(off);
        for (uint32_t e = 0; e < in.n_edges; e++) {
            t1.push_back((unsigned)off + in.edge_i[e]);
            t2.push_back((unsigned)off + in.edge_j[e]);
            for (int k = 0; k < 3; k++) {
                meas.push_back(in.meas[3 * (size_t)e + k]);
                info.push_back(std::exp(in.log_w[3 * (size_t)e + k]) * in.lambda);
            }
        }
        memcpy(poses.data() + 3 * (size_t)off, in.poses, 3 * (size_t)in.n_poses * sizeof(double));
        anchor_rows.push_back(off);
        anchor_vals.push_back(in.anchor);
        diag_rows.push_back(off);
        for (int r = off + (int)in.n_poses; r < off + padded; r++) {
            diag_rows.push_back(r);
            anchor_rows.push_back(r);
            anchor_vals.push_back(1.0);
        }
    }
    DevMem &m = g->mem;
    if (dupload(m, g->st, &g->d_poses, poses) != cudaSuccess || dupload(m, g->st, &g->d_ei, t1) != cudaSuccess ||
        dupload(m, g->st, &g->d_ej, t2) != cudaSuccess || dupload(m, g->st, &g->d_meas, meas) != cudaSuccess ||
        dupload(m, g->st, &g->d_info, info) != cudaSuccess) {
        gslam_set_last_error("upload failed");
        return fail(GSLAM_ERR_CUDA);
    }
    rc = finish_setup(g, t1, t2, &diag_rows, &segments);
    if (rc != GSLAM_OK) return fail(rc);
    std::vector<int64_t> slots(anchor_rows.size());
    for (size_t a = 0; a < anchor_rows.size(); a++) slots[a] = g->S.diag_slot[g->S.iperm[anchor_rows[a]]];
    B.n_anchor = (int)slots.size();
    if (dupload(m, g->st, &B.d_anchor_slots, slots) != cudaSuccess ||
        dupload(m, g->st, &B.d_anchor_vals, anchor_vals) != cudaSuccess ||
        dupload(m, g->st, &B.d_pose_off, B.pose_off) != cudaSuccess ||
        dupload(m, g->st, &B.d_n_real, B.n_real) != cudaSuccess ||
        dalloc(m, &B.d_gdiff, (size_t)n_graphs) != cudaSuccess || dalloc(m, &B.d_res, (size_t)n_graphs) != cudaSuccess ||
        dalloc(m, &B.d_chunk_part, (size_t)n_graphs * B.max_chunks) != cudaSuccess ||
        dalloc(m, &B.d_active, 1) != cudaSuccess ||
        cudaMallocHost(&B.h_res, n_graphs * sizeof(PcgResult)) != cudaSuccess ||
        cudaMallocHost(&B.h_gdiff, n_graphs * sizeof(double)) != cudaSuccess) {
        gslam_set_last_error("batch buffers");
        return fail(GSLAM_ERR_CUDA);
    }
    rc = batch_partition(g);
    if (rc == GSLAM_OK && !g->o.disable_resident) rc = batch_clusters_build(g, g->o.precision == GSLAM_PREC_MIXED);
    if (rc != GSLAM_OK) return fail(rc);
    if (cudaStreamSynchronize(g->st) != cudaSuccess) { gslam_set_last_error("setup failed"); return fail(GSLAM_ERR_CUDA); }
    *out = g;
    return GSLAM_OK;
}

/*
 * Whether a batch's graphs get a thread-block cluster each (pcg_cluster.cu), and of how many
 * CTAs: if all of them fit 16 (20,480 rows at most) and that is the faster way by the
 * estimates, else the grid-wide solver takes the whole batch.
 * The GPU is shared by all graphs at once, and few full CTAs use it
 * better than many sparse ones, so each takes the smallest cluster with 20 slices per CTA in
 * FP64, 40 in FP32 (about what shared memory holds), or 16 CTAs. Ms of solve per round, 64
 * graphs of 500 to 17,000 poses, 10 / 20 / 30 / 40 slices: FP64 14.3 / 10.3 / 11.4 / 11.9, FP32
 * - / 8.4 / 8.1 / 7.7 (8.9 and 6.7 since the sums are shorter); the grid-wide batch solver takes
 * 23.8 and 15.8; cluster sizes that are no power of two, 40 slices per CTA for the smaller
 * graphs alone, or higher stream priorities for larger graphs, gain nothing. While twice as many
 * CTAs still run at once, every cluster is doubled, down to four slices per CTA. Launches
 * of equal cluster shape run side by side on their own streams, the largest clusters first,
 * and the GPU starts the next cluster as one ends; the graphs of a launch come in order of
 * falling size, so the last to start are short.
 * A batch is not split between the two: the grid-wide solver's iteration is mostly barriers and the
 * widest row's chain of loads, so it takes almost as long for a part of the batch as for all
 * of it. Us per iteration, clusters and then a graph of 25,000 poses / all grid-wide: with 20
 * graphs of 500 poses 17.3 / 15.2, 8 of 20,000 48.7 / 40.2; two graphs of 15,000 poses with 2
 * random closures per pose, one of which fits no cluster, 48.6 / 26.7.
 */
/* SMs that a cluster takes out of use: so many run at once that the others' SMs stay empty */
static double cluster_sms(int ctas, int n_sm) {
    return ctas == 16 ? n_sm / 7.0 : ctas == 8 ? n_sm / 15.0 : ctas == 4 ? n_sm / 33.0 : (double)ctas;
}

static int batch_clusters_build(gslam_graph *g, bool fp32) {
    BatchState &B = *g->batch;
    BatchClusters &K = B.clusters[fp32 ? 1 : 0];
    if (K.built) return GSLAM_OK;
    const gslam_structure &S = g->S;
    const int G = B.n_graphs, elem = fp32 ? 4 : 8;
    K.launches.clear();
    int max_ctas = GSLAM_CLUSTER_CTAS;
    for (int shape = 0; shape < 4; shape++)
        if (GSLAM_BATCH_SHAPES >> shape & 1) max_ctas = std::min(max_ctas, pcg_cluster_ctas(fp32, true, shape, GSLAM_CLUSTER_CTAS, GSLAM_RES_SMEM_MAX));
    std::vector<gslam_cluster_part> part(G);
    std::vector<int> lcol(S.n_slots, 0), keep(S.n_slices, 0), pos(S.n_slices, 0), ctas(G, 0);
    auto first = [&](int q) { return B.pose_off[q] / 32; };
    auto plan = [&](int q, int c) {
        return gslam_cluster_plan(S, first(q), first(q + 1), c, GSLAM_BATCH_SHAPES, elem, GSLAM_RES_SMEM_MAX, &part[q], &lcol, &keep, &pos);
    };
    int64_t used = 0;
    for (int q = 0; q < G; q++) {
        const int ns = first(q + 1) - first(q);
        int c = 1;
        const int per = fp32 ? GSLAM_CLUSTER_SLICES : GSLAM_CLUSTER_SLICES / 2;
        while (c < max_ctas && c * per < ns) c *= 2;
        for (; c <= max_ctas; c *= 2)
            if (plan(q, c)) { ctas[q] = c; break; }
        if (ctas[q] == 0) { K.built = true; return GSLAM_OK; }
        used += ctas[q];
    }
    for (bool more = true; more && 2 * used <= g->L.n_sm;) {
        more = false;
        for (int q = 0; q < G; q++)
            if (2 * ctas[q] <= max_ctas && 8 * ctas[q] <= first(q + 1) - first(q)) {
                used += ctas[q];
                ctas[q] *= 2;
                more = true;
            }
    }
    std::vector<int> order(G);
    double longest = 0.0, sm_us = 0.0, sms = 0.0;
    for (int q = 0; q < G; q++) {
        /* a doubled cluster that does not fit after all (longer halos) is halved again */
        if (part[q].ctas != ctas[q])
            while (!plan(q, ctas[q])) ctas[q] /= 2;
        order[q] = q;
        const double us = gslam_cluster_us(part[q], elem), n = cluster_sms(ctas[q], g->L.n_sm);
        longest = std::max(longest, us);
        sms += n;
        sm_us += n * us;
    }
    /* at most what list scheduling needs; 0.9: no change of solver at a tie */
    const double us = sms <= g->L.n_sm ? longest : sm_us / g->L.n_sm + longest;
    if (us > 0.9 * gslam_batch_us(S.max_width, S.n_slots / 32, elem)) { K.built = true; return GSLAM_OK; }
    /* launches: cluster size and CTA shape */
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        if (part[a].ctas != part[b].ctas) return part[a].ctas > part[b].ctas;
        if (part[a].shape != part[b].shape) return part[a].shape > part[b].shape;
        return first(a + 1) - first(a) > first(b + 1) - first(b);
    });
    std::vector<ClusterJob> jobs;
    std::vector<int> bounds, halo, exp_ptr;
    std::vector<unsigned> exp;
    for (size_t i = 0; i < order.size(); i++) {
        const int q = order[i];
        const gslam_cluster_part &p = part[q];
        const int prev = i ? order[i - 1] : -1;
        if (prev < 0 || part[prev].ctas != p.ctas || part[prev].shape != p.shape)
            K.launches.push_back({ (int)i, 0, p.ctas, 0, p.shape, 0 });
        BatchClusters::Launch &l = K.launches.back();
        l.n_jobs++;
        l.threads = std::max(l.threads, p.threads);
        l.smem = std::max(l.smem, p.smem);
        jobs.push_back({ q, first(q), first(q + 1) - first(q), (int)halo.size(), (int)bounds.size(), (int)exp_ptr.size(),
                         p.halo_max });
        bounds.insert(bounds.end(), p.bounds.begin(), p.bounds.end());
        halo.insert(halo.end(), p.n_halo.begin(), p.n_halo.end());
        for (int e : p.exp_ptr) exp_ptr.push_back(e + (int)exp.size());
        exp.insert(exp.end(), p.exp.begin(), p.exp.end());
    }
    for (const BatchClusters::Launch &l : K.launches)
        if (l.ctas == 1 && pcg_cluster_ctas(fp32, true, l.shape, 1, GSLAM_RES_SMEM_MAX) == 0) {
            K.launches.clear();
            K.built = true;
            return GSLAM_OK;
        }
    DevMem &m = g->mem;
    CK(dupload_all(m, g->st, { dpart(&K.d_jobs, jobs), dpart(&K.d_bounds, bounds), dpart(&K.d_halo, halo),
                               dpart(&K.d_lcol, lcol), dpart(&K.d_keep, keep), dpart(&K.d_pos, pos),
                               dpart(&K.d_exp_ptr, exp_ptr), dpart(&K.d_exp, exp) }));
    if (!B.fork) CK(cudaEventCreateWithFlags(&B.fork, cudaEventDisableTiming));
    while (B.side.size() < K.launches.size()) {
        cudaStream_t t;
        cudaEvent_t e;
        CK(cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking));
        B.side.push_back(t);
        CK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        B.side_done.push_back(e);
    }
    K.built = true;
    return GSLAM_OK;
}

/* Solves the batch's systems on the handle's stream, in clusters or with the grid-wide solver.
 * skip (may be null) marks graphs to leave alone. */
static int batch_launch(gslam_graph *g, const PcgParams &P, BatchParams BP, bool fp32, const std::vector<int> *skip) {
    BatchState &B = *g->batch;
    cudaStream_t st = g->st;
    BatchClusters &K = B.clusters[fp32 ? 1 : 0];
    const int G = B.n_graphs;
    /* the test hook names a CTA of the grid-wide solver */
    const bool clusters = g->o.test_absent_cta < 0 && !g->o.disable_resident;
    if (clusters) {
        const int rc = batch_clusters_build(g, fp32);
        if (rc != GSLAM_OK) return rc;
    }
    if (skip) {
        if (!B.d_skip) CK(dalloc(g->mem, &B.d_skip, (size_t)G));
        CK(cudaMemcpyAsync(B.d_skip, skip->data(), (size_t)G * sizeof(int), cudaMemcpyHostToDevice, st));
        BP.skip = B.d_skip;
    }
    if (!clusters || K.launches.empty()) {
        CK(launch_pcg_batch(st, P, BP, B.grid, B.block, B.smem_bytes, fp32));
        return GSLAM_OK;
    }
    ClusterParams Q;
    memset(&Q, 0, sizeof Q);
    Q.jobs = K.d_jobs;
    Q.cta_slice = K.d_bounds;
    Q.n_halo = K.d_halo;
    Q.lcol = K.d_lcol;
    Q.keep = K.d_keep;
    Q.pos = K.d_pos;
    Q.exp_ptr = K.d_exp_ptr;
    Q.exp = K.d_exp;
    Q.slice_ptr = P.slice_ptr;
    Q.row_len = P.row_len;
    Q.n_rows = P.n_rows;
    Q.val = P.val;
    Q.val32 = P.val32;
    Q.dinv = P.dinv;
    Q.b4 = P.b4;
    Q.x4 = P.x4;
    Q.bf4 = BP.bf4;
    Q.xf4 = P.xf4;
    Q.tol_rel = P.tol_rel;
    Q.max_iter = P.max_iter;
    Q.spin_limit = P.spin_limit;
    Q.absent_cta = -1;
    Q.smem_budget = GSLAM_RES_SMEM_MAX;
    Q.res = P.res;
    Q.gres = BP.res;
    Q.skip = BP.skip;
    Q.cap = BP.cap;
    CK(cudaEventRecord(B.fork, st));
    for (size_t i = 0; i < K.launches.size(); i++) {
        const BatchClusters::Launch &l = K.launches[i];
        CK(cudaStreamWaitEvent(B.side[i], B.fork, 0));
        Q.job0 = l.job0;
        Q.ctas = l.ctas;
        CK(launch_pcg_cluster(B.side[i], Q, l.n_jobs, l.threads, l.shape, l.smem, fp32, true));
        CK(cudaEventRecord(B.side_done[i], B.side[i]));
    }
    for (size_t i = 0; i < K.launches.size(); i++) CK(cudaStreamWaitEvent(st, B.side_done[i], 0));
    return GSLAM_OK;
}

static int batch_solve_mixed(gslam_graph *g, gslam_solve_stats *per_graph, gslam_solve_stats *total);

int batch_solve(gslam_graph *g, gslam_solve_stats *per_graph, gslam_solve_stats *total, const std::vector<int> *skip) {
    if (g->o.precision == GSLAM_PREC_MIXED) return batch_solve_mixed(g, per_graph, total);
    BatchState &B = *g->batch;
    DevLayout *L = &g->L;
    cudaStream_t st = g->st;
    launch_diag_inv(st, L->n_rows, L->diag_slot, L->val, L->dinv);
    CK(cudaGetLastError());
    PcgParams P;
    memset(&P, 0, sizeof P);
    P.n_rows = L->n_rows;
    P.n_slices = L->n_slices;
    P.slice_ptr = L->slice_ptr;
    P.row_len = L->row_len;
    P.col = L->col;
    P.val = L->val;
    P.dinv = L->dinv;
    P.b4 = L->b4;
    P.x4 = L->x4; P.r4 = L->r4; P.z4 = L->z4; P.p4a = L->p4a; P.p4b = L->p4b; P.q4 = L->q4;
    P.tol_rel = g->o.tol;
    P.max_iter = g->o.max_iter;
    P.gs = L->gs;
    P.res = L->res;
    const double ms = g->o.barrier_timeout_ms > 0 ? g->o.barrier_timeout_ms : 2000.0;
    P.spin_limit = (long long)(ms * (double)L->clock_khz);
    P.absent_cta = g->o.test_absent_cta;
    if (2.0 * (double)std::max(g->o.max_iter, 0) * B.grid + 8.0 * B.grid >= 4294967295.0) {
        gslam_set_last_error("max_iter too large for the solver's 32-bit barrier counter");
        return GSLAM_ERR_TOO_LARGE;
    }
    BatchParams BP;
    memset(&BP, 0, sizeof BP);
    BP.n_graphs = B.n_graphs;
    BP.cta_slice = B.d_cta_slice;
    BP.slice_graph = B.d_slice_graph;
    BP.cta_g0 = B.d_cta_g0;
    BP.cta_g1 = B.d_cta_g1;
    BP.graph_cta0 = B.d_graph_cta0;
    BP.graph_ncta = B.d_graph_ncta;
    BP.part_off = B.d_part_off;
    BP.total_parts = B.total_parts;
    BP.partials = B.d_partials;
    BP.res = B.d_res;
    BP.active = B.d_active;
    CK(cudaMemsetAsync(L->gs, 0, sizeof(GridSync), st));
    CK(cudaMemsetAsync(L->res, 0, sizeof(PcgResult), st));
    CK(cudaMemsetAsync(B.d_res, 0, B.n_graphs * sizeof(PcgResult), st));
    CK(cudaMemcpyAsync(B.d_active, &B.n_graphs, sizeof(int), cudaMemcpyHostToDevice, st));
    CK(record_event(L->ev0, st));
    const int rc = batch_launch(g, P, BP, false, skip);
    if (rc != GSLAM_OK) return rc;
    CK(record_event(L->ev1, st));
    CK(cudaMemcpyAsync(g->h_res, L->res, sizeof(PcgResult), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(B.h_res, B.d_res, B.n_graphs * sizeof(PcgResult), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    float solve_ms = 0.f;
    solve_ms = elapsed_ms(L->ev0, L->ev1);
    gslam_solve_stats agg;
    memset(&agg, 0, sizeof agg);
    agg.solve_ms = solve_ms;
    for (int q = 0; q < B.n_graphs; q++) {
        const PcgResult &r = B.h_res[q];
        const double rel = r.bnorm > 0 ? r.rnorm / r.bnorm : 0.0;
        if (per_graph) {
            memset(&per_graph[q], 0, sizeof per_graph[q]);
            per_graph[q].iterations = r.iterations;
            per_graph[q].reason = r.reason;
            per_graph[q].rel_residual = rel;
            per_graph[q].solve_ms = solve_ms;
        }
        agg.iterations = std::max(agg.iterations, r.iterations);
        agg.rel_residual = std::max(agg.rel_residual, rel);
        if (r.reason != GSLAM_STOP_TOL) agg.reason = r.reason;
    }
    if (total) *total = agg;
    if (g->h_res->timeout) {
        gslam_set_last_error("solver barrier wait timed out");
        return GSLAM_ERR_DEVICE_TIMEOUT;
    }
    return GSLAM_OK;
}

/*
 * Mixed-precision batch: iterative refinement driven from the host, every graph at
 * once. Per step: the FP32 right-hand side (the FP64 residual, 0 for graphs already
 * done), one launch of the batched PCG in FP32 (FP32 values and vectors, FP64 D^-1 and
 * dot products, per-graph scalars, inner tolerance inner_tol, each graph capped by what
 * is left of its max_iter), x += d in FP64, and the FP64 residual b - A x with per-graph
 * norms. A graph stops at tol, at max_iter inner iterations, or when a whole inner pass
 * (not one cut short by what is left of max_iter) did not halve the graph's residual
 * (stagnation); the graphs that stagnate are solved again in FP64 and those results are
 * reported.
 */
static int batch_solve_mixed(gslam_graph *g, gslam_solve_stats *per_graph, gslam_solve_stats *total) {
    BatchState &B = *g->batch;
    DevLayout *L = &g->L;
    cudaStream_t st = g->st;
    DevMem &m = g->mem;
    const int G = B.n_graphs;
    int rc = gslam_layout_ensure_fp32(L, st);
    if (rc != GSLAM_OK) return rc;
    if (!L->val32_fresh) {
        launch_val_to_f32(st, 9 * L->n_slots, L->val, L->val32);
        L->val32_fresh = true;
    }
    if (!B.d_bf4) {
        CK(dalloc(m, &B.d_bf4, 4 * 32 * (size_t)L->n_slices));
        CK(dalloc(m, &B.d_gactive, (size_t)G));
        CK(dalloc(m, &B.d_gcap, (size_t)G));
        CK(dalloc(m, &B.d_gres, (size_t)G));
        CK(cudaMallocHost(&B.h_gres, G * sizeof(double)));
    }
    launch_diag_inv(st, L->n_rows, L->diag_slot, L->val, L->dinv);
    /* x = 0; r = b - A 0 = b with per-graph ||b|| */
    CK(cudaMemsetAsync(L->x4, 0, 4 * 32 * (size_t)L->n_slices * sizeof(double), st));
    CK(cudaMemsetAsync(L->q4, 0, 4 * 32 * (size_t)L->n_slices * sizeof(double), st));
    launch_batch_resid(st, G, B.d_pose_off, L->b4, L->q4, L->r4, B.d_gres, B.d_chunk_part, B.max_chunks);
    CK(cudaMemcpyAsync(B.h_gres, B.d_gres, G * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    std::vector<double> bnorm(G), rel(G, 1.0);
    std::vector<int> its(G, 0), refs(G, 0), reason(G, GSLAM_STOP_MAXIT), active(G, 1), cap(G, 0);
    bool stagnated = false;
    for (int q = 0; q < G; q++) {
        bnorm[q] = std::sqrt(B.h_gres[q]);
        if (bnorm[q] == 0.0) { active[q] = 0; reason[q] = GSLAM_STOP_TOL; rel[q] = 0.0; }
    }
    PcgParams P;
    memset(&P, 0, sizeof P);
    P.n_rows = L->n_rows;
    P.n_slices = L->n_slices;
    P.slice_ptr = L->slice_ptr;
    P.row_len = L->row_len;
    P.col = L->col;
    P.val32 = L->val32;
    P.dinv = L->dinv;
    P.xf4 = L->f[0]; P.rf4 = L->f[1]; P.zf4 = L->f[2]; P.pfa4 = L->f[3]; P.pfb4 = L->f[4]; P.qf4 = L->f[5];
    P.tol_rel = g->o.inner_tol;
    P.gs = L->gs;
    P.res = L->res;
    const double ms_lim = g->o.barrier_timeout_ms > 0 ? g->o.barrier_timeout_ms : 2000.0;
    P.spin_limit = (long long)(ms_lim * (double)L->clock_khz);
    P.absent_cta = g->o.test_absent_cta;
    BatchParams BP;
    memset(&BP, 0, sizeof BP);
    BP.n_graphs = G;
    BP.cta_slice = B.d_cta_slice;
    BP.slice_graph = B.d_slice_graph;
    BP.cta_g0 = B.d_cta_g0;
    BP.cta_g1 = B.d_cta_g1;
    BP.graph_cta0 = B.d_graph_cta0;
    BP.graph_ncta = B.d_graph_ncta;
    BP.part_off = B.d_part_off;
    BP.total_parts = B.total_parts;
    BP.partials = B.d_partials;
    BP.res = B.d_res;
    BP.active = B.d_active;
    BP.bf4 = B.d_bf4;
    BP.cap = B.d_gcap;
    CK(record_event(L->ev0, st));
    for (int step = 0; step < std::max(g->o.max_refine, 1); step++) {
        /* each graph's inner pass is capped by what is left of its own budget */
        int n_active = 0, cap_max = 0;
        for (int q = 0; q < G; q++) {
            if (!active[q]) { cap[q] = 0; continue; }
            cap[q] = std::min(g->o.inner_max_iter, g->o.max_iter - its[q]);
            if (cap[q] <= 0) { active[q] = 0; reason[q] = GSLAM_STOP_MAXIT; continue; }
            n_active++;
            cap_max = std::max(cap_max, cap[q]);
        }
        if (n_active == 0) break;
        P.max_iter = cap_max;
        CK(cudaMemcpyAsync(B.d_gactive, active.data(), G * sizeof(int), cudaMemcpyHostToDevice, st));
        CK(cudaMemcpyAsync(B.d_gcap, cap.data(), G * sizeof(int), cudaMemcpyHostToDevice, st));
        launch_batch_rhs32(st, L->n_rows, B.d_slice_graph, B.d_gactive, L->r4, B.d_bf4);
        CK(cudaMemsetAsync(L->gs, 0, sizeof(GridSync), st));
        CK(cudaMemsetAsync(L->res, 0, sizeof(PcgResult), st));
        CK(cudaMemsetAsync(B.d_res, 0, G * sizeof(PcgResult), st));
        CK(cudaMemcpyAsync(B.d_active, &G, sizeof(int), cudaMemcpyHostToDevice, st));
        rc = batch_launch(g, P, BP, true, nullptr);
        if (rc != GSLAM_OK) return rc;
        launch_batch_add_x(st, L->n_rows, L->f[0], L->x4);
        launch_spmv64(st, L->n_rows, L->n_slices, L->slice_ptr, L->row_len, L->col, L->val, L->x4, L->q4);
        launch_batch_resid(st, G, B.d_pose_off, L->b4, L->q4, L->r4, B.d_gres, B.d_chunk_part, B.max_chunks);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(g->h_res, L->res, sizeof(PcgResult), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(B.h_res, B.d_res, G * sizeof(PcgResult), cudaMemcpyDeviceToHost, st));
        CK(cudaMemcpyAsync(B.h_gres, B.d_gres, G * sizeof(double), cudaMemcpyDeviceToHost, st));
        CK(cudaStreamSynchronize(st));
        if (g->h_res->timeout) {
            gslam_set_last_error("solver barrier wait timed out");
            return GSLAM_ERR_DEVICE_TIMEOUT;
        }
        for (int q = 0; q < G; q++) {
            if (!active[q]) continue;
            its[q] += B.h_res[q].iterations;
            refs[q]++;
            const double prev = rel[q];
            rel[q] = std::sqrt(B.h_gres[q]) / bnorm[q];
            if (rel[q] < g->o.tol) { active[q] = 0; reason[q] = GSLAM_STOP_TOL; }
            else if (its[q] >= g->o.max_iter || refs[q] >= g->o.max_refine) { active[q] = 0; reason[q] = GSLAM_STOP_MAXIT; }
            else if (rel[q] > 0.5 * prev && !(B.h_res[q].reason == GSLAM_STOP_MAXIT && cap[q] < g->o.inner_max_iter)) {
                /* a whole inner pass (to its tolerance or its inner_max_iter) did not halve the
                 * FP64 residual: FP32 cannot resolve this graph. A pass cut short by what was
                 * left of the graph's max_iter is not this. */
                active[q] = 0;
                reason[q] = GSLAM_STOP_STAGNATION;
                stagnated = true;
            }
        }
    }
    CK(record_event(L->ev1, st));
    CK(cudaEventSynchronize(L->ev1));
    float solve_ms = 0.f;
    solve_ms = elapsed_ms(L->ev0, L->ev1);
    if (stagnated) {
        /* the FP32 inner solves cannot resolve these graphs: solve just them again in FP64
         * (from x = 0, the reference's start); every other graph keeps its mixed solution */
        std::vector<int> skip(G);
        for (int q = 0; q < G; q++) skip[q] = reason[q] == GSLAM_STOP_STAGNATION ? 0 : 1;
        std::vector<gslam_solve_stats> s64(G);
        gslam_solve_stats tot64;
        gslam_opts keep = g->o;
        g->o.precision = GSLAM_PREC_FP64;
        rc = batch_solve(g, s64.data(), &tot64, &skip);
        g->o = keep;
        if (rc != GSLAM_OK) return rc;
        for (int q = 0; q < G; q++)
            if (!skip[q]) {
                its[q] += s64[q].iterations;
                refs[q] = -refs[q];
                reason[q] = s64[q].reason;
                rel[q] = s64[q].rel_residual;
            }
        solve_ms += (float)tot64.solve_ms;
    }
    gslam_solve_stats agg;
    memset(&agg, 0, sizeof agg);
    agg.solve_ms = solve_ms;
    for (int q = 0; q < G; q++) {
        if (per_graph) {
            memset(&per_graph[q], 0, sizeof per_graph[q]);
            per_graph[q].iterations = its[q];
            per_graph[q].refinements = refs[q];
            per_graph[q].reason = reason[q];
            per_graph[q].rel_residual = rel[q];
            per_graph[q].solve_ms = solve_ms;
        }
        agg.iterations = std::max(agg.iterations, its[q]);
        agg.refinements = std::max(agg.refinements, refs[q]);
        agg.rel_residual = std::max(agg.rel_residual, rel[q]);
        if (reason[q] != GSLAM_STOP_TOL) agg.reason = reason[q];
    }
    if (total) *total = agg;
    return GSLAM_OK;
}

int gslam_batch_round(gslam_graph *g, gslam_solve_stats *per_graph) {
    if (!g || !g->batch) BAD("not a batch");
    BatchState &B = *g->batch;
    if (!g->ev_round0) {
        CK(cudaEventCreate(&g->ev_round0));
        CK(cudaEventCreate(&g->ev_round1));
    }
    CK(record_event(g->ev_round0, g->st));
    int rc = gslam_linearise(g);
    if (rc != GSLAM_OK) return rc;
    rc = gslam_assemble(g);
    if (rc != GSLAM_OK) return rc;
    rc = batch_solve(g, per_graph, nullptr);
    if (rc != GSLAM_OK) return rc;
    launch_pose_update(g->st, g->n_poses, g->L.iperm, g->L.x4, g->d_poses, g->d_dx, g->o.angle_wrap,
                       g->d_block_sums, g->n_upd_blocks, g->d_diff);
    launch_batch_diff(g->st, B.n_graphs, B.d_pose_off, B.d_n_real, g->d_dx, B.d_gdiff, B.d_chunk_part, B.max_chunks);
    CK(cudaGetLastError());
    CK(record_event(g->ev_round1, g->st));
    CK(cudaMemcpyAsync(B.h_gdiff, B.d_gdiff, B.n_graphs * sizeof(double), cudaMemcpyDeviceToHost, g->st));
    CK(cudaStreamSynchronize(g->st));
    float ms = 0.f;
    ms = elapsed_ms(g->ev_round0, g->ev_round1);
    if (per_graph)
        for (int q = 0; q < B.n_graphs; q++) {
            per_graph[q].diff = B.h_gdiff[q];
            per_graph[q].round_ms = ms;
        }
    return GSLAM_OK;
}

int gslam_batch_layout(gslam_graph *g, uint32_t *n_graphs, uint32_t *pose_offset) {
    if (!g || !g->batch || !n_graphs) BAD("not a batch");
    *n_graphs = (uint32_t)g->batch->n_graphs;
    if (pose_offset)
        for (int q = 0; q <= g->batch->n_graphs; q++) pose_offset[q] = (uint32_t)g->batch->pose_off[q];
    return GSLAM_OK;
}

int gslam_batch_in_clusters(const gslam_graph *g, int *yes) {
    if (!g || !g->batch || !yes) BAD("not a batch");
    const BatchClusters &K = g->batch->clusters[g->o.precision == GSLAM_PREC_MIXED ? 1 : 0];
    *yes = g->o.test_absent_cta < 0 && !g->o.disable_resident && !K.launches.empty();
    return GSLAM_OK;
}

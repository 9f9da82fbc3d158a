/* gslam_api_internal.h — device-side objects behind the C ABI (internal). */
#ifndef GSLAM_API_INTERNAL_H
#define GSLAM_API_INTERNAL_H

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <initializer_list>
#include <string>
#include <vector>

#include "gslam.h"
#include "gslam_internal.h"
#include "kernels.cuh"

/* Device allocations owned by one object, released together. */
struct DevMem {
    std::vector<void *> ptrs;
    void release();
};

/* Device copy of a layout plus the solver's work vectors. */
struct DevLayout {
    DevMem mem;
    int n_rows = 0, n_slices = 0;
    int64_t n_slots = 0;
    int *perm = nullptr, *iperm = nullptr, *row_len = nullptr, *col = nullptr;
    int *diag_slot = nullptr, *chunk_slice = nullptr;
    int64_t *slice_ptr = nullptr, *slot_csr = nullptr;
    double *val = nullptr, *dinv = nullptr;
    float *val32 = nullptr;
    bool val32_fresh = false;      /* val32 holds the current values */
    double *b4 = nullptr, *x4 = nullptr, *r4 = nullptr, *z4 = nullptr;
    double *p4a = nullptr, *p4b = nullptr, *q4 = nullptr;
    float *f[6] = { nullptr, nullptr, nullptr, nullptr, nullptr, nullptr };
    double *partials = nullptr;
    GridSync *gs = nullptr;        /* followed by the tagged reductions' slots (tag_words) */
    size_t tag_bytes = 0;
    PcgResult *res = nullptr;
    int grid = 0, block = 0, n_sm = 0;
    int clock_khz = 2000000;       /* SM clock, for barrier wait limits */
    int partial_capacity = 0;
    /* shared-memory-resident solver (pcg_resident.cu), when the layout fits */
    bool resident = false;
    int res_grid = 0;
    int res_slices = 0;            /* slices of the CTA that owns most */
    /* per slice: block positions in shared memory, and where (FP64 resident, mixed, one-reduction) */
    int *res_keep = nullptr, *res_pos = nullptr, *mixed_keep = nullptr, *mixed_pos = nullptr, *cg_keep = nullptr,
        *cg_pos = nullptr;
    int *cta_slice = nullptr;      /* [res_grid + 1] */
    int *lcol = nullptr, *halo_ptr = nullptr, *halo_rows = nullptr; /* CTA-local columns, halo lists */
    unsigned char *row_export = nullptr; /* rows some other CTA's halo lists */
    /* mixed and one-reduction: some CTA's halo does not fit its shared memory; v of those rows
     * (made on first use, n_halo rows) */
    bool long_halo = false;
    int n_halo = 0;
    double *halo_v = nullptr;
    size_t smem_bytes = 0;
    bool mixed_ok = false;          /* the mixed solver's shared-memory layout fits */
    size_t mixed_smem_bytes = 0;   /* dynamic shared memory per launch: the largest CTA layout (mixed_smem_layout) */
    bool cg_ok = false;             /* the FP64 one-reduction solver's layout fits */
    size_t cg_smem_bytes = 0;
    /* cluster solver (pcg_cluster.cu), when the graph fits one thread-block cluster */
    bool cluster_ok = false;
    int cluster_ctas = 0, cluster_threads = 0, cluster_shape = 0, cluster_vctas = 0;
    size_t cluster_smem = 0;
    ClusterJob *cluster_job = nullptr;
    int *cluster_bounds = nullptr, *cluster_halo = nullptr, *cluster_lcol = nullptr, *cluster_exp_ptr = nullptr;
    int *cluster_keep = nullptr, *cluster_pos = nullptr;
    unsigned *cluster_exp = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;   /* brackets the solver launch */
    int max_grid_alloc() const { return partial_capacity; }
};

/* A batch solved in one cluster per graph (pcg_cluster.cu), in one precision: launches of equal
 * cluster shape, largest clusters first; none when the grid-wide solver takes the batch. */
struct BatchClusters {
    struct Launch {
        int job0, n_jobs, ctas, threads, shape;
        size_t smem;
    };
    bool built = false;
    std::vector<Launch> launches;
    ClusterJob *d_jobs = nullptr;
    int *d_bounds = nullptr, *d_halo = nullptr, *d_lcol = nullptr, *d_exp_ptr = nullptr;
    int *d_keep = nullptr, *d_pos = nullptr;
    unsigned *d_exp = nullptr;
};

/* A batch of independent SE(2) graphs as one block-diagonal graph (batch.cu). */
struct BatchState {
    int n_graphs = 0;
    std::vector<int> pose_off;   /* [n_graphs + 1] first (padded) pose of each graph */
    std::vector<int> n_real;     /* [n_graphs] poses of each graph without padding */
    int *d_pose_off = nullptr, *d_n_real = nullptr;
    int n_anchor = 0;
    int64_t *d_anchor_slots = nullptr;
    double *d_anchor_vals = nullptr;
    /* solver partition */
    int grid = 0, block = 0, max_slices = 0;
    size_t smem_bytes = 0;
    int total_parts = 0;
    int *d_cta_slice = nullptr, *d_slice_graph = nullptr, *d_cta_g0 = nullptr, *d_cta_g1 = nullptr;
    int *d_graph_cta0 = nullptr, *d_graph_ncta = nullptr, *d_part_off = nullptr;
    double *d_partials = nullptr, *d_gdiff = nullptr;
    PcgResult *d_res = nullptr, *h_res = nullptr;
    double *h_gdiff = nullptr;
    int *d_active = nullptr;
    /* mixed batches: FP32 right-hand side, per-graph active flags and residual norms */
    float *d_bf4 = nullptr;
    int *d_gactive = nullptr;
    int *d_gcap = nullptr;       /* mixed: each graph's iteration cap for the current inner pass */
    double *d_gres = nullptr, *h_gres = nullptr;
    BatchClusters clusters[2];   /* FP64, FP32 */
    std::vector<cudaStream_t> side; /* the launches' streams, and their fork and join events */
    std::vector<cudaEvent_t> side_done;
    cudaEvent_t fork = nullptr;
    int *d_skip = nullptr;       /* [n_graphs] graphs the FP64 rerun of a stagnated mixed batch leaves alone */
    /* chunk sums of the per-graph norm kernels */
    double *d_chunk_part = nullptr;
    int max_chunks = 1;
};

struct gslam_graph {
    int device = 0;
    cudaStream_t st = nullptr;
    gslam_opts o;
    int factors = GSLAM_FACTORS_REFERENCE;
    gslam_structure S;
    DevLayout L;
    DevMem mem;
    int n_poses = 0;
    int64_t n_obs_edges = 0, n_edges = 0;
    double delta = 1.0, lambda = 1.0, mns[4] = { 0.19, 0.001, 0.13, 0.2 };
    double anchor = 1000000.0;
    /* reference factor inputs */
    double *d_poses = nullptr, *d_controls = nullptr, *d_z_rb = nullptr;
    unsigned *d_z_step = nullptr, *d_pj = nullptr, *d_pk = nullptr;
    /* SE(2) factor inputs */
    unsigned *d_ei = nullptr, *d_ej = nullptr;
    double *d_meas = nullptr, *d_info = nullptr; /* info = exp(log_w) */
    /* per-round buffers */
    double *d_blocks = nullptr;
    int64_t *d_ctr_ptr = nullptr, *d_ctr = nullptr, *d_xi_ptr = nullptr, *d_xi_ctr = nullptr;
    double *d_dx = nullptr, *d_block_sums = nullptr, *d_diff = nullptr;
    int n_upd_blocks = 1;
    double *d_csr_tmp = nullptr, *d_xi_tmp = nullptr;
    double *d_adj = nullptr;   /* adjoint: rhs, mu (3 N each), per-edge gradient (3 E) */
    BatchState *batch = nullptr; /* non-null for a batch of graphs */
    /* landmark groups of the z list (reference graphs) */
    std::vector<unsigned> lm_ids;
    int64_t *d_lm_ptr = nullptr;
    unsigned *d_lm_members = nullptr;
    double *d_lm_ms = nullptr;
    PcgResult *h_res = nullptr;
    double *h_diff = nullptr;
    /* round cost: per-edge terms, block sums, total (allocated on first use) */
    double *d_edge_cost = nullptr, *d_cost_blocks = nullptr, *d_cost = nullptr;
    PcgResult last_res = {};
    cudaEvent_t ev_round0 = nullptr, ev_round1 = nullptr;
    /* gslam_opts.round_graph: the captured round and how many rounds ran eagerly */
    cudaGraphExec_t round_exec = nullptr;
    int eager_rounds = 0;
};

/* batch: a batch's layout, which the single-graph resident solvers never run on */
int gslam_layout_upload(DevLayout *L, const gslam_structure &S, cudaStream_t st, int device,
                        const gslam_opts &o, bool batch = false);
int gslam_layout_ensure_fp32(DevLayout *L, cudaStream_t st);
/* grid_order: the dot products are added in the grid-wide solver's order (a cluster of one
 * CTA keeps it, a larger one is not used), for systems that may be indefinite, where CG
 * amplifies rounding */
int gslam_layout_solve(DevLayout *L, cudaStream_t st, const gslam_opts &o, PcgResult *h_res,
                       gslam_solve_stats *stats, bool grid_order = false);
void gslam_layout_release(DevLayout *L);
/* Assembles Omega / xi from edge blocks; optionally also writes the reference's CSR
 * values (csr_vals) and xi in original order (xi_orig), both device pointers. */
int gslam_assemble_ex(gslam_graph *g, const double *blocks, double *csr_vals, double *xi_orig);
/* gslam_update that also records `done` (may be null) after the update kernels. */
int gslam_update_ex(gslam_graph *g, double *diff, cudaEvent_t done);
/* Records an error message for gslam_last_error(). */
void gslam_set_last_error(const char *msg);
void gslam_set_error(const char *fmt, const char *what, int code);

/* ---- helpers shared by the handle API's translation units (api.cu, batch_api.cu) ---- */

/* a failing CUDA call: record it for gslam_last_error() and return GSLAM_ERR_CUDA */
#define CK(call)                                                                               \
    do {                                                                                       \
        cudaError_t _e = (call);                                                               \
        if (_e != cudaSuccess) {                                                               \
            gslam_set_last_error((std::string(#call) + ": " + cudaGetErrorString(_e)).c_str()); \
            return GSLAM_ERR_CUDA;                                                             \
        }                                                                                      \
    } while (0)

#define BAD(msg)                        \
    do {                                \
        gslam_set_last_error(msg);      \
        return GSLAM_ERR_BAD_INPUT;     \
    } while (0)

/* device allocation owned by m (released with it) */
template <class T>
inline cudaError_t dalloc(DevMem &m, T **p, size_t n) {
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, (n ? n : 1) * sizeof(T));
    if (e != cudaSuccess) return e;
    m.ptrs.push_back(q);
    *p = (T *)q;
    return cudaSuccess;
}

/* device copy of a host vector, owned by m */
template <class T>
inline cudaError_t dupload(DevMem &m, cudaStream_t st, T **p, const std::vector<T> &v) {
    cudaError_t e = dalloc(m, p, v.size());
    if (e != cudaSuccess) return e;
    if (v.empty()) return cudaSuccess;
    return cudaMemcpyAsync(*p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, st);
}

/* device copies of several host vectors in one allocation, each from a 256-byte boundary: an
 * allocation costs 0.1 ms on an idle host and milliseconds on a busy one */
struct DevPart {
    void **p;
    const void *v;
    size_t bytes;
};
template <class T>
inline DevPart dpart(T **p, const std::vector<T> &v) { return DevPart{ (void **)p, v.data(), v.size() * sizeof(T) }; }
inline cudaError_t dupload_all(DevMem &m, cudaStream_t st, std::initializer_list<DevPart> parts) {
    size_t end = 0;
    for (const DevPart &q : parts) end += (q.bytes + 255) / 256 * 256;
    std::vector<unsigned char> all(end);
    unsigned char *base = nullptr;
    cudaError_t e = dalloc(m, &base, end);
    if (e != cudaSuccess) return e;
    end = 0;
    for (const DevPart &q : parts) {
        if (q.bytes) memcpy(all.data() + end, q.v, q.bytes);
        *q.p = base + end;
        end += (q.bytes + 255) / 256 * 256;
    }
    return all.empty() ? cudaSuccess : cudaMemcpyAsync(base, all.data(), all.size(), cudaMemcpyHostToDevice, st);
}

/* an event record that a stream capture keeps as a node of the graph */
cudaError_t record_event(cudaEvent_t e, cudaStream_t st);
/* elapsed time between two recorded events, 0 when unavailable */
float elapsed_ms(cudaEvent_t a, cudaEvent_t b);
/* creation steps every handle shares: options, device, stream, pinned status words */
int common_setup(gslam_graph *g, const gslam_opts *opts);
/* structure, layout upload and per-round buffers of a handle with edges (t1, t2) */
int finish_setup(gslam_graph *g, const std::vector<unsigned> &t1, const std::vector<unsigned> &t2,
                 const std::vector<int> *diag_rows = nullptr, const std::vector<int> *segments = nullptr);
/* the batched solve behind gslam_solve / gslam_round on a batch handle (batch_api.cu) */
int batch_solve(gslam_graph *g, gslam_solve_stats *per_graph, gslam_solve_stats *total,
                const std::vector<int> *skip = nullptr);

#endif
